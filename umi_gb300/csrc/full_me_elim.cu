// Full-search motion estimation of 16x16 blocks by exact elimination.
//
// Same operator as full_me.cu (main/full_me.cu:8-64: SAD of a block of `cur`
// against `ref` at every displacement, reference pixels clamped to the frame;
// argmin first in raster order of (dy, dx), main/full_me.cu:70-71) with the
// same result for every input, but most candidates are ruled out by a lower
// bound instead of being summed (successive elimination, Li & Salari 1995,
// here over sixteen 4x4 cells per block).  With S a cell's pixel sum and
// q = floor(S / 16),
//   SAD >= sum over cells |S_cur - S_ref| >= sum (16 |q_cur - q_ref| - 15) = 16 C - 240,
// C = sum |q_cur - q_ref|: four `vabsdiff4` per candidate instead of 64.  The
// candidate of least C is summed exactly; with U its SAD, only candidates with
// 16 C - 240 <= U can reach the minimum (or tie with it), and only those are
// summed: about 30 of 4225 at +-32 on the benchmark's frame pairs, 170 on a
// panning camera.  Where more are left (unrelated frames: a sixth), whole columns
// of eleven rows that hold one are summed; where a cell's mean says no more than
// its neighbours' (noise; told from the first two blocks' pixels) every candidate
// is, without the bound.
//
// What bounds it: the integer ALU pipe (the bound's `vabsdiff4`, the cells'
// byte permutations, the exact sums) and issue.  One CTA serves a run of NB
// horizontally adjacent blocks (their windows overlap, so the cells of the run's
// window are formed once), one block when the blocks come from a list or are
// moved by centres:
//   0. the window's pixels to shared memory (rows and columns clamped);
//   1. cells: lane = 16 columns x 3 rows; every position x stores the word of
//      its four cells x, x + 4, x + 8, x + 12, so that a candidate's cell row
//      is one aligned word;
//   2. bound: thread = (block, column, up to 66 rows): 45 cell words streamed
//      once per 33 rows against the block's four cell rows, the costs kept in
//      registers (two of 12 bits per word);
//   3. the least C of each block; its exact SAD, by every warp for itself;
//   4. the survivors' list, from the costs still in registers;
//   5. exact SADs of the survivors, eight lanes of two rows per candidate;
//      blocks with too many survivors: thread = (column, group of rows).
// Everything is shared memory and barriers: no workspace, no waits on other
// CTAs.
//
// Measured on a GB300 (graph replays, ms), every candidate summed by a
// warp-specialised kernel -> here: 1080p +-32, blocks moved one by one 0.148 ->
// 0.0405, panning camera 0.148 -> 0.046, unrelated frames 0.148 -> 0.119, noise
// 0.148 -> 0.155; +-64 0.580 -> 0.202, unrelated 0.52, noise 0.585; +-16 (by the
// general kernel) 0.087 -> 0.0225, 0.051, 0.054; 4K +-64 2.19 -> 0.74, noise 2.29.
// Noise costs up to 7 % (4K, +-32) where the windows were fetched ahead by warps of
// their own.  At 86 % of the ALU pipe it is bound by that.  By phase at 1080p +-32:
// pixels 12 us, cells 8, bound 14, survivors 5, exact sums 5.  Tried: two blocks per
// run on 160 threads (0.058 ms), three on 224 (0.047), six cell rows per lane
// (0.048), a persistent form with the next run's pixels in flight (0.051), noise
// left to a second, warp-specialised launch (0.055 with noise at 0.173), two to four
// neighbouring runs per CTA, the later ones without the bound after a hard one
// (0.045, panning camera 0.070).
#include <algorithm>

#include "common.h"

namespace {

constexpr int RC = 33;       // candidate rows per pass of the bound, two passes per thread
// SW: words per window row, an odd number of 16-byte pieces for 16 nb + 2 r
// pixels; QS: words per row of the cell words, the columns of a run's window, a
// multiple of 4; THREADS: at most, for a column each.
struct Wide {
	static constexpr int SW = 36, QS = 132, THREADS = 288;
};
// One block, +-32 at most: lists, centres and frames with too few runs.  A third of
// Wide's shared memory, so that seven CTAs fit (1080p with centres, +-32: 99 us, 157
// with Wide; 256 x 448, +-32: 14.6 and 17.0).
struct Narrow {
	static constexpr int SW = 20, QS = 68, THREADS = 128;
};
constexpr int MAXT = Wide::THREADS;
constexpr int MAXNB = 8;
constexpr int NC = MAXNB / 2;     // cells of a run per lane
constexpr size_t kSmemThree = 74 * 1024;  // dynamic shared memory that leaves room for three CTAs per SM
constexpr int CR = 3;        // cell rows per lane and step
constexpr int GA = 17, GB = 22;  // candidate rows per thread of the search of every candidate
constexpr int GS = 11;           // and where rows without a survivor are left out (8: 6 % slower)

__device__ __forceinline__ uint32_t sad4(uint32_t a, uint32_t b, uint32_t c) {
	uint32_t d;
	asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
	return d;
}
__device__ __forceinline__ void copy4(uint32_t* dst, const void* src) {
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void copy16(uint32_t* dst, const void* src) {
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
	uint32_t d;
	asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
	return d;
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
	uint32_t d;
	asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
	return d;
}

// n / d for 0 <= n < 2^31 by multiply and shift (Granlund & Montgomery 1994).
struct Div {
	uint32_t mul;
	int shift;
	static Div by(int d) {
		int l = 0;
		while (((int64_t)1 << l) < d) ++l;
		const uint64_t num = (uint64_t)1 << (31 + l);
		return {(uint32_t)((num + (uint64_t)d - 1) / (uint64_t)d), 31 + l};
	}
	__device__ __forceinline__ int operator()(int n) const { return (int)(((uint64_t)(uint32_t)n * mul) >> shift); }
};

// The same in 32 bits for n d < 2^22 and n / d < 2^10: indices below nd * nd <= 129^2.
struct SmallDiv {
	uint32_t mul;
	static SmallDiv by(int d) { return {(uint32_t)(((1 << 22) + d - 1) / d)}; }
	__device__ __forceinline__ int operator()(int n) const { return (int)(((uint32_t)n * mul) >> 22); }
};

struct ElimArgs {
	const uint8_t* cur;
	const uint8_t* ref;
	const int32_t* centers;     // optional: per-block search centres (cy, cx)
	int32_t* out;               // (nblk, 3): mv_y, mv_x, sad
	const int32_t* list;        // optional: search only these blocks (slot i -> block list[i])
	const int32_t* list_count;  // number of valid slots of `list` (device word)
	int h, w, r, nd, nbx, slots;
	int nb;                     // blocks per run (1 with a list or centres)
	int runs_x, units;          // runs per block row; runs in all (slots with a list or centres)
	int nchunk;                 // threads per column, two passes of RC rows each (one when nd <= RC)
	int wrows, wwords;          // window: rows, words per row
	int qrows, ncols, spw;      // cells: rows, columns; row pieces a warp forms at a time
	int pieces;                 // 16-byte pieces per window row
	int limit;                  // survivors a block may keep before it is searched exhaustively
	int rows;                   // of every candidate's search: GA or GB
	int cols;                   // columns of the exhaustive search in tasks, the others one by one
	int tasks;                  // of the exhaustive search, per block
	int cur_words;              // cur's rows are 4-byte aligned
	int ref_pieces;             // ref's rows are 16-byte aligned
	int cur_pieces;             // cur's rows are 16-byte aligned
	Div div_x;                  // by blocks or runs per block row
	SmallDiv div_nd, div_task, div_piece, div_spw, div_tasks, div_cols;  // by nd, nd * nchunk, pieces, spw, tasks, cols
	uint32_t mul16, mul64k;     // 16 and 2^16 (runtime values: the keys stay multiply-adds, off the ALU pipe)
	// shared memory offsets in words
	int copy, o_copy;           // stride and start of the shifted windows (over the cell words)
	int o_task;                 // tasks of the exhaustive search (over the cell words too)
	int team_words;             // shared memory of a team
	int o_q, o_blk, o_cell, o_list;
};

// Four pixels gx .. gx + 3 of row `row` (offset `off` of the frame's first
// pixel), columns clamped to the frame.
__device__ __forceinline__ uint32_t pixels4(const uint8_t* __restrict__ frame, size_t off, int gx, int w) {
	const uint8_t* row = frame + off;
	uint32_t v = 0;
#pragma unroll
	for (int t = 0; t < 4; ++t) v |= (uint32_t)__ldg(row + min(max(gx + t, 0), w - 1)) << (8 * t);
	return v;
}

// SADs of G candidate rows of one column against the block: the least, as
// sad * 32 + row (of the first `rows`, where they are fewer).  p: the column's words, shifted so that they
// start on a word.  One word of the rows at a time: a ring of G window words
// meets each block row, so the registers hold G sums and G words, and the SADs
// need 0.15 loads each and no address arithmetic.
template <int G, int SW>
__device__ __forceinline__ uint32_t exhaustive_rows(const uint32_t* __restrict__ p, const uint32_t* __restrict__ blk,
                                                    int rows) {
	uint32_t acc[G];
#pragma unroll
	for (int q = 0; q < G; ++q) acc[q] = 0;
#pragma unroll 1
	for (int k = 0; k < 4; ++k, ++p, ++blk) {
		uint32_t ring[G];
#pragma unroll
		for (int q = 0; q < G - 1; ++q) ring[q] = p[q * SW];
#pragma unroll
		for (int py = 0; py < 16; ++py) {
			const uint32_t c = blk[4 * py];
			ring[(py + G - 1) % G] = p[(py + G - 1) * SW];
#pragma unroll
			for (int q = 0; q < G; ++q) acc[q] = sad4(c, ring[(py + q) % G], acc[q]);
		}
	}
	if (rows < G)  // a range below eight
#pragma unroll
		for (int q = 1; q < G; ++q)
			if (q >= rows) acc[q] = 1u << 26;
	uint32_t k = acc[0] * 32u;
#pragma unroll
	for (int q = 1; q < G; ++q) k = min(k, acc[q] * 32u + (uint32_t)q);
	return k;
}

// Costs of rows y0 .. y0 + RC - 1 of one column (col: the shared address of
// cell row y0), packed: p[i] = cost[i] | cost[i + 16] << 16, p16 = cost[32].
// Returns the least cost * 64 + row (the first row among equals).
template <int QS>
__device__ __forceinline__ uint32_t bound_rows(unsigned col, const uint32_t (&c)[4], int rows, uint32_t mul16,
                                               uint32_t mul64k, uint32_t (&p)[16], uint32_t& p16) {
	uint32_t cost[RC];
#pragma unroll
	for (int y = 0; y < RC + 12; ++y) {
		uint32_t v;  // volatile: hoisted loads would push the costs out of the registers
		asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(col + 4u * QS * y));
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			const int k = y - 4 * i;
			if (k >= 0 && k < RC) cost[k] = sad4(c[i], v, i == 0 ? 0u : cost[k]);
		}
	}
	if (rows < RC)  // a range below 33 rows
#pragma unroll
		for (int i = 0; i < RC; ++i)
			if (i >= rows) cost[i] = 4095u;  // above every cost (at most 16 * 255), within 12 bits
	// 16-bit keys cost * 16 + row, formed by multiply-adds (off the ALU pipe)
	uint32_t m = 0xffffffffu;
#pragma unroll
	for (int i = 0; i < 16; ++i) {
		p[i] = cost[i + 16] * mul64k + cost[i];
		m = min_u16x2(m, p[i] * mul16 + ((uint32_t)i | ((uint32_t)i << 16)));
	}
	p16 = cost[32];
	const uint32_t lo = m & 0xffffu, hi = m >> 16;
	return min(min(((lo >> 4) << 6) | (lo & 15u), ((hi >> 4) << 6) | 16u | (hi & 15u)), (cost[32] << 6) | 32u);
}

// Bit i: row i (0 .. 31) of the packed costs is at most T (12 bits each).
__device__ __forceinline__ uint32_t survivors(const uint32_t (&p)[16], uint32_t T) {
	const uint32_t t2 = (T | (T << 16)) + 0x80008000u;
	uint32_t m = 0;
#pragma unroll
	for (int i = 0; i < 16; ++i) m = (m >> 1) | ((t2 - p[i]) & 0x80008000u);
	return m;
}

// A run of horizontally adjacent blocks (or one block).
struct Run {
	int blk0, bx0, by, nb, cy, cx;
};
template <bool LIST>
__device__ __forceinline__ Run run_of(const ElimArgs& a, int unit) {
	Run u{0, 0, 0, 1, 0, 0};
	if (LIST || a.centers) {
		u.blk0 = LIST ? a.list[unit] : unit;
		u.by = a.div_x(u.blk0);
		u.bx0 = u.blk0 - u.by * a.nbx;
		if (a.centers) {
			u.cy = a.centers[2 * u.blk0];
			u.cx = a.centers[2 * u.blk0 + 1];
		}
	} else {
		u.by = a.div_x(unit);
		u.bx0 = (unit - u.by * a.runs_x) * a.nb;
		u.nb = min(a.nb, a.nbx - u.bx0);
		u.blk0 = u.by * a.nbx + u.bx0;
	}
	return u;
}

// A run's window and blocks into shared memory, cp.async where the source is
// aligned (words past the last block's window are loaded but not used).
template <int SW>
__device__ __forceinline__ void load_run(const ElimArgs& a, const Run& u, uint32_t* win, uint32_t* blkw, int row0,
                                         int piece, int piece_rows, int tid, int nt) {
	const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
	const int gy0 = 16 * u.by + u.cy - a.r, gx0 = 16 * u.bx0 + u.cx - a.r;
	if (a.ref_pieces && (gx0 & 15) == 0 && gx0 >= 0 && gx0 + 16 * a.pieces <= a.w) {
		const uint8_t* src = a.ref + gx0 + 16 * piece;
		for (int row = row0; row < a.wrows; row += piece_rows)
			copy16(win + row * SW + 4 * piece, src + (size_t)min(max(gy0 + row, 0), a.h - 1) * a.w);
	} else {
		const size_t total = (size_t)a.h * a.w;
		for (int row = warp; row < a.wrows; row += nwarps) {
			const size_t off = (size_t)min(max(gy0 + row, 0), a.h - 1) * a.w;
			for (int k = lane; k < a.wwords; k += 32) {
				const int gx = gx0 + 4 * k;
				uint32_t* dst = win + row * SW + k;
				const size_t o = off + gx;
				const uintptr_t p = reinterpret_cast<uintptr_t>(a.ref) + o;
				if (gx < 0 || gx + 4 > a.w) {
					*dst = pixels4(a.ref, off, gx, a.w);
				} else if ((p & 3) == 0) {
					copy4(dst, a.ref + o);
				} else if (o >= 4 && o + 8 <= total) {  // two aligned words of the frame
					const uint32_t* s = reinterpret_cast<const uint32_t*>(p & ~(uintptr_t)3);
					*dst = __funnelshift_r(__ldg(s), __ldg(s + 1), 8 * (int)(p & 3));
				} else {
					*dst = pixels4(a.ref, off, gx, a.w);
				}
			}
		}
	}
	if (a.cur_pieces) {
		for (int i = tid; i < 16 * u.nb; i += nt) {
			const int b = i >> 4, row = i & 15;
			copy16(blkw + 4 * i, a.cur + (size_t)(16 * u.by + row) * a.w + 16 * (u.bx0 + b));
		}
		return;
	}
	for (int i = tid; i < 64 * u.nb; i += nt) {
		const int b = i >> 6, row = (i >> 2) & 15, k = i & 3;
		const size_t off = (size_t)(16 * u.by + row) * a.w;
		const int gx = 16 * (u.bx0 + b) + 4 * k;
		if (a.cur_words) copy4(blkw + i, a.cur + off + gx);
		else blkw[i] = pixels4(a.cur, off, gx, a.w);
	}
}

// Cell words of rows y0 .. y0 + CR - 1 (those below qrows) and the 16 columns
// of group g (columns 16 g .. 16 g + cols - 1 are stored).  Sums are 16-bit
// pairs: down four rows in pixel order, then regrouped so that the pair
// members are eight columns apart (ev: columns j, j + 8; od: j + 4, j + 12),
// which makes the four sums across sliding additions, the byte packing three
// instructions per word and the words of columns x + 4, + 8, + 12 byte shifts.
// The next group's columns come from lane + spw (the last group's are not
// needed: it holds the window's last 16 columns).
// Sums are clamped to [lo, lo + 2^s * 256) and stored as (sum - lo) >> s.
template <int SW, int QS>
__device__ __forceinline__ void form_cells(const ElimArgs& a, const uint32_t* __restrict__ win, uint32_t* __restrict__ q,
                                           int y0, int g, int cols, uint32_t lo, int sh) {
	const uint32_t lo2 = lo * 0x10001u, hi2 = lo2 + ((256u << sh) - 1u) * 0x10001u;
	const uint32_t* src = win + y0 * SW + 4 * g;
	uint32_t ring[3][8], sum[8];
	auto row = [&](uint32_t (&v)[8]) {
		const uint4 x = *reinterpret_cast<const uint4*>(src);
		src += SW;
		const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			v[2 * k] = w[k] & 0x00ff00ffu;                    // columns 4k, 4k + 2
			v[2 * k + 1] = __byte_perm(w[k], 0u, 0x4341);     // columns 4k + 1, 4k + 3
		}
	};
#pragma unroll
	for (int i = 0; i < 3; ++i) row(ring[i]);
#pragma unroll
	for (int k = 0; k < 8; ++k) sum[k] = ring[0][k] + ring[1][k] + ring[2][k];
	uint32_t* dst = q + y0 * QS + 16 * g;
#pragma unroll
	for (int i = 0; i < CR; ++i) {
		uint32_t n[8], V[8], ev[4], od[4];
		row(n);
#pragma unroll
		for (int k = 0; k < 8; ++k) {
			V[k] = sum[k] + n[k];
			sum[k] = V[k] - ring[i % 3][k];
			ring[i % 3][k] = n[k];
		}
		ev[0] = __byte_perm(V[0], V[4], 0x5410); ev[2] = __byte_perm(V[0], V[4], 0x7632);
		ev[1] = __byte_perm(V[1], V[5], 0x5410); ev[3] = __byte_perm(V[1], V[5], 0x7632);
		od[0] = __byte_perm(V[2], V[6], 0x5410); od[2] = __byte_perm(V[2], V[6], 0x7632);
		od[1] = __byte_perm(V[3], V[7], 0x5410); od[3] = __byte_perm(V[3], V[7], 0x7632);
		uint32_t te = (ev[0] + ev[1] + ev[2]) + ev[3], to = (od[0] + od[1] + od[2]) + od[3], B[4], N[4];
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const uint32_t ce = min_u16x2(max_u16x2(te, lo2), hi2) - lo2, co = min_u16x2(max_u16x2(to, lo2), hi2) - lo2;
			B[j] = ((ce >> sh) & 0x00ff00ffu) | ((co << (8 - sh)) & 0xff00ff00u);
			if (j < 3) {
				te = te - ev[j] + od[j];
				to = to - od[j] + __byte_perm(ev[j], __shfl_down_sync(0xffffffffu, ev[j], a.spw), 0x5432);
			}
			N[j] = __shfl_down_sync(0xffffffffu, B[j], a.spw);
		}
		if (y0 + i < a.qrows) {
			if (cols > 0) *reinterpret_cast<uint4*>(dst) = make_uint4(B[0], B[1], B[2], B[3]);
#pragma unroll
			for (int m = 1; m < 4; ++m)
				if (4 * m < cols) {
					const uint32_t sel = m == 1 ? 0x4321u : m == 2 ? 0x5432u : 0x6543u;
					*reinterpret_cast<uint4*>(dst + 4 * m) =
						make_uint4(__byte_perm(B[0], N[0], sel), __byte_perm(B[1], N[1], sel), __byte_perm(B[2], N[2], sel),
					               __byte_perm(B[3], N[3], sel));
				}
		}
		dst += QS;
	}
}

// Exact SAD of a candidate of block b by eight lanes (sub 0 .. 7), two rows each.
template <int SW>
__device__ __forceinline__ void exact_sum(const ElimArgs& a, const uint32_t* win, const uint32_t* blkw, uint32_t* best,
                                          int b, int iy, int ix, int sub) {
	const int X = 16 * b + ix;
	const uint32_t* w = win + (iy + sub) * SW + (X >> 2);
	const uint4* cr = reinterpret_cast<const uint4*>(blkw + b * 64) + sub;
	const uint32_t sel = 0x3210u + 0x1111u * (uint32_t)(X & 3);
	uint32_t s = 0;
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		const uint4 c = cr[8 * h];
		uint32_t v[5];
#pragma unroll
		for (int k = 0; k < 5; ++k) v[k] = w[8 * h * SW + k];
		s = sad4(c.x, __byte_perm(v[0], v[1], sel), s);
		s = sad4(c.y, __byte_perm(v[1], v[2], sel), s);
		s = sad4(c.z, __byte_perm(v[2], v[3], sel), s);
		s = sad4(c.w, __byte_perm(v[3], v[4], sel), s);
	}
#pragma unroll
	for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	if (sub == 0) atomicMin(&best[b], (s << 15) | (uint32_t)(iy * a.nd + ix));
}

// A whole warp's keys into their blocks' least.
__device__ __forceinline__ void least_of(uint32_t* best, int b, uint32_t key, int lane) {
	if (__all_sync(0xffffffffu, b == __shfl_sync(0xffffffffu, b, 0))) {
		const uint32_t least = __reduce_min_sync(0xffffffffu, key);
		if (lane == 0) atomicMin(&best[b], least);
	} else {
		atomicMin(&best[b], key);
	}
}

// Exact SADs of `count` tasks (block, group of G rows, column), one per thread, by
// the warps that make as many for each of the SM's four schedulers (a ninth would
// keep one of them busy half as long again).
template <int G, int SW>
__device__ __forceinline__ void exhaustive(const ElimArgs& a, const uint32_t* tasks, int count, const uint32_t* win,
                                           const uint32_t* copies, const uint32_t* blkw, uint32_t* best, int tid, int nt) {
	const int lane = tid & 31, nw = nt >= 128 ? nt & ~127 : nt;
	if (tid >= nw) return;
	for (int t0 = tid - lane; t0 < count; t0 += nw) {  // warp-uniform
		const uint32_t e = tasks[min(t0 + lane, count - 1)];  // lanes past the end repeat the last task
		const int b = (int)(e >> 16), ix = (int)(e & 255u), iy = max(min((int)(e >> 8 & 255u) * G, a.nd - G), 0);
		const uint32_t* w = (ix & 3 ? copies + ((ix & 3) - 1) * a.copy : win) + iy * SW + ((16 * b + ix) >> 2);
		const uint32_t s = exhaustive_rows<G, SW>(w, blkw + b * 64, a.nd);
		const uint32_t key = ((s >> 5) << 15) | (uint32_t)((iy + (int)(s & 31u)) * a.nd + ix);
		least_of(best, b, key, lane);
	}
}

// Whether one of the rows s .. s + n - 1 is a survivor: bit i of m row i, e row 32.
__device__ __forceinline__ bool any_row(uint32_t m, bool e, int s, int n) {
	const uint64_t v = m | ((uint64_t)e << 32), rows = ((uint64_t)1 << n) - 1;
	return s <= -n || s > 32 ? false : (v & (s >= 0 ? rows << s : rows >> -s)) != 0;
}

// MINB: CTAs per SM (three at 72 registers; two where shared memory holds no
// more; seven of Narrow).  TEAMS 0: a run per CTA.  Otherwise a list of blocks,
// whose length only the GPU knows: with no more blocks than CTAs a CTA takes a
// block with all its threads, beyond that it works as TEAMS teams with a block
// each, of a share of the threads and shared memory, that never wait for one
// another.  (Fallback list of 130 blocks at 1080p, +-64, most of them hard: the pass
// around it 79 us with two CTAs per SM, 68 so; 28 000 blocks at 4K: 1.17 ms with all
// threads on each block, 0.91 so.)
template <class W, int MINB, int TEAMS>
__global__ void __launch_bounds__(W::THREADS * (TEAMS ? TEAMS : 1), MINB) full_me_elim_kernel(const ElimArgs a) {
	constexpr int SW = W::SW, QS = W::QS, NT = W::THREADS, N = TEAMS ? TEAMS : 1;
	constexpr bool LIST = TEAMS > 0;
	extern __shared__ __align__(16) uint32_t smem[];
	__shared__ uint32_t seeds[N][MAXNB], bests[N][MAXNB];
	__shared__ int cnts[N][MAXNB], totals[N], tasks[N];
	int units = a.units;
	if (LIST) units = min(units, *a.list_count);
	const bool teams = LIST && units > (int)gridDim.x;
	const int team = teams ? (int)threadIdx.x / NT : 0, nteams = teams ? N : 1;
	const int tid = (int)threadIdx.x - team * NT, nt = teams ? NT : (int)blockDim.x;
	const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
	auto sync = [&] {  // the threads of this team
		if (LIST) asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(nt) : "memory");
		else __syncthreads();
	};
	uint32_t *seed = seeds[team], *best = bests[team];
	int *cnt = cnts[team], &total_cnt = totals[team], &n_tasks = tasks[team];
	uint32_t* sm = smem + team * a.team_words;
	uint32_t* win = sm;              // [wrows][sw]
	uint32_t* q = sm + a.o_q;        // [max(nd, RC) + 12][QS]: cell words
	uint32_t* blkw = sm + a.o_blk;   // [nb][16][4]
	uint32_t* cell = sm + a.o_cell;  // [nb][4]
	uint32_t* list = sm + a.o_list;  // [nb * limit]: block, row, column
	const int nd = a.nd, r = a.r;
	// this thread's column of the bound and its rows: two passes from iy0, the
	// second one ending with row iy1 + RC - 1 (passes and threads overlap where
	// the rows do not divide)
	const int tb = a.div_task(tid), tt = tid - tb * nd * a.nchunk, tc = a.div_nd(tt), tx = tt - tc * nd;
	const int iy0 = min(2 * RC * tc, max(0, nd - RC)), iy1 = min(iy0 + RC, max(0, nd - RC));
	const int wb0 = a.div_task(tid - lane), wb1 = a.div_task(tid - lane + 31);  // the blocks of this warp's columns
	const int gl = a.div_spw(lane), seg = lane - gl * a.spw;
	const int prow = a.div_piece(tid), piece = tid - prow * a.pieces;
	const int piece_rows = nt / a.pieces, row0 = prow < piece_rows ? prow : a.wrows;

	for (int unit = blockIdx.x * nteams + team; unit < units; unit += gridDim.x * nteams) {
		const Run u = run_of<LIST>(a, unit);
		load_run<SW>(a, u, win, blkw, row0, piece, piece_rows, tid, nt);
		if (tid < MAXNB) {
			seed[tid] = 0xffffffffu;
			best[tid] = 0xffffffffu;
			cnt[tid] = 0;
		}
		if (tid == 0) total_cnt = n_tasks = 0;
		asm volatile("cp.async.wait_all;" ::: "memory");
		sync();
		// ---- 1. cells: cur's, by every warp for the scale and, from the first two
		// blocks, for whether the bound can serve; then the window's
		uint32_t sums[NC], mn = 0xffffffffu, mx = 0, differ = 0;
#pragma unroll
		for (int t = 0; t < NC; ++t) {
			if (32 * t >= 16 * u.nb) break;
			const int i = min(lane + 32 * t, 16 * u.nb - 1);
			const uint32_t* px = blkw + (i >> 4) * 64 + ((i >> 2) & 3) * 16 + (i & 3);
			uint32_t v = 0, w[4];
#pragma unroll
			for (int k = 0; k < 4; ++k) {
				w[k] = px[4 * k];
				v = sad4(w[k], 0u, v);
			}
			if (t == 0) {  // cells' differences with their neighbours (eighths) and pixels' with those below (quarters)
				const uint32_t l = __shfl_xor_sync(0xffffffffu, v, 1), o = __shfl_xor_sync(0xffffffffu, v, 4);
				const uint32_t cells = max(v, l) - min(v, l) + max(v, o) - min(v, o);
				const uint32_t pixels = sad4(w[0], w[1], sad4(w[1], w[2], sad4(w[2], w[3], 0u)));
				differ = __reduce_add_sync(0xffffffffu, lane < 16 * u.nb ? (cells >> 3) << 16 | pixels >> 2 : 0u);
			}
			sums[t] = v;
			mn = min(mn, v);
			mx = max(mx, v);
		}
		mn = __reduce_min_sync(0xffffffffu, mn);
		mx = __reduce_max_sync(0xffffffffu, mx);
		int hard = (1 << u.nb) - 1, count = -1;  // blocks and tasks of the exhaustive search (all of them)
		// A list with few small windows is done soonest without the bound (130 blocks,
		// +-32: 10 us whatever their content, else 9 to 14).  Elsewhere cells' sums that
		// differ less from their neighbours' than 1.25 times the pixels from those below
		// are noise: a random block stays below that in 999 of 1000 cases, one of the
		// benchmark's texture (sigma 5.6, with noise of 2) above it.  Not so blocks at the
		// frame's edges; in a list of a few rounds one of them, summed in full, would
		// outlast the others, so shorter ones of wide windows go by the bound (the
		// coarse pass at 4K, 8 pairs: 136.6 us, 134.5 so).
		const bool alone = LIST && !teams && NT == Narrow::THREADS;
		const bool tell = !LIST || NT == Narrow::THREADS || units > 4 * nteams * (int)gridDim.x;
		if (!alone && (!tell || 8 * (differ >> 16) >= 5 * (differ & 0xffffu))) {
			hard = 0;
			int sh = 2;
			while (sh < 4 && (256u << sh) < 2 * (mx - mn)) ++sh;
			const uint32_t half = 128u << sh, mid = (mn + mx) >> 1, lo = mid > half ? mid - half : 0u;
			if (warp == 0) {
#pragma unroll
				for (int t = 0; t < NC; ++t)
					if (lane + 32 * t < 16 * u.nb)
						reinterpret_cast<uint8_t*>(cell)[lane + 32 * t] =
							(uint8_t)((min(max(sums[t], lo), lo + (256u << sh) - 1u) - lo) >> sh);
			}
			// lane = (group gl of 16 columns, piece `seg` of CR rows)
			for (int s0 = warp * a.spw; s0 * CR < a.qrows; s0 += nwarps * a.spw)
				form_cells<SW, QS>(a, win, q, (s0 + seg) * CR, min(gl, a.pieces - 1), gl < a.pieces ? a.ncols - 16 * gl : 0, lo, sh);
			sync();
			// ---- 2. bound
			const bool task = tb < u.nb;
			uint32_t p0[16], p1[16], l0 = 0, l1 = 0, k0 = 0xffffffffu, k1 = 0xffffffffu;
			if (task) {
				uint32_t c[4];
#pragma unroll
				for (int i = 0; i < 4; ++i) c[i] = cell[4 * tb + i];
				const unsigned col = (unsigned)__cvta_generic_to_shared(q + 16 * tb + tx);
				k0 = bound_rows<QS>(col + 4u * QS * iy0, c, nd - iy0, a.mul16, a.mul64k, p0, l0);
				if (nd > RC) k1 = bound_rows<QS>(col + 4u * QS * iy1, c, RC, a.mul16, a.mul64k, p1, l1);
			}
			// ---- 3. the least C of each block
			const uint32_t key = min(((k0 >> 6) << 15) | (uint32_t)((iy0 + (int)(k0 & 63u)) * nd + tx),
			                         ((k1 >> 6) << 15) | (uint32_t)((iy1 + (int)(k1 & 63u)) * nd + tx));
			if (wb0 == wb1) {
				const uint32_t m = __reduce_min_sync(0xffffffffu, task ? key : 0xffffffffu);
				if (lane == 0 && m != 0xffffffffu) atomicMin(&seed[tb], m);
			} else if (task) {
				atomicMin(&seed[tb], key);
			}
			sync();
			int T = -1;
			for (int b = wb0; b <= min(wb1, u.nb - 1); ++b) {
				const uint32_t idx = seed[b] & 0x7fffu;
				const int iy = a.div_nd((int)idx), X = 16 * b + (int)idx - iy * nd + 8 * (lane & 1);
				const uint32_t* w = win + (iy + (lane >> 1)) * SW + (X >> 2);
				const uint32_t sel = 0x3210u + 0x1111u * (uint32_t)(X & 3);
				const uint2 c = *reinterpret_cast<const uint2*>(blkw + b * 64 + 2 * lane);
				const uint32_t w1 = w[1];
				const uint32_t s = sad4(c.x, __byte_perm(w[0], w1, sel), sad4(c.y, __byte_perm(w1, w[2], sel), 0u));
				const uint32_t U = __reduce_add_sync(0xffffffffu, s);
				if (lane == 0) atomicMin(&best[b], (U << 15) | idx);
				// an exact match: the seed, the first candidate of cost 0, is also the first exact one
				if (b == tb && U != 0) T = (int)min((U + (16u << sh) - 16u) >> sh, 4095u);
			}
			// ---- 4. survivors
			uint32_t m0 = 0, m1 = 0;
			bool e0 = false, e1 = false;
			if (task && (int)(min(k0, k1) >> 6) <= T) {
				if ((int)(k0 >> 6) <= T) {
					m0 = survivors(p0, (uint32_t)T);
					if (nd < RC) m0 &= 0xffffffffu >> (32 - nd);
					e0 = nd >= RC && (int)l0 <= T;
				}
				if ((int)(k1 >> 6) <= T) {
					m1 = survivors(p1, (uint32_t)T);
					e1 = (int)l1 <= T;
				}
				const int n = __popc(m0) + __popc(m1) + e0 + e1;
				if (atomicAdd(&cnt[tb], n) + n <= a.limit) {
					uint32_t* dst = list + atomicAdd(&total_cnt, n);
					const uint32_t e = ((uint32_t)tb << 16) | (uint32_t)tx;
					if (e0) *dst++ = e + ((uint32_t)(iy0 + 32) << 8);
					if (e1) *dst++ = e + ((uint32_t)(iy1 + 32) << 8);
					for (uint32_t m = m0; m; m &= m - 1) *dst++ = e + ((uint32_t)(iy0 + __ffs((int)m) - 1) << 8);
					for (uint32_t m = m1; m; m &= m - 1) *dst++ = e + ((uint32_t)(iy1 + __ffs((int)m) - 1) << 8);
				}
			}
			sync();
			// ---- 5. exact sums
			for (int b = 0; b < u.nb; ++b) hard |= (cnt[b] > a.limit) << b;
			const int n = hard == (1 << u.nb) - 1 ? 0 : total_cnt, sub = lane & 7;
			for (int j0 = 4 * warp; j0 < n; j0 += 4 * nwarps) {
				const uint32_t e = list[min(j0 + (lane >> 3), n - 1)];  // lanes past the end repeat the last candidate
				const int b = (int)(e >> 16);
				if (hard && __all_sync(0xffffffffu, hard >> b & 1)) continue;  // listed before its block had too many
				exact_sum<SW>(a, win, blkw, best, b, (int)(e >> 8 & 255u), (int)(e & 255u), sub);
			}
			if (hard) {  // uniform over the team: the tasks that hold a survivor
				const bool mine = task && (hard >> tb & 1);
#pragma unroll 1
				for (int g = 0; g * GS < nd; ++g) {
					const int y = max(min(g * GS, nd - GS), 0);
					const bool any = mine && y + GS > 2 * RC * tc && (any_row(m0, e0, y - iy0, GS) || any_row(m1, e1, y - iy1, GS));
					const uint32_t lanes = __ballot_sync(0xffffffffu, any);
					int at = 0;
					if (lane == 0 && lanes) at = atomicAdd(&n_tasks, __popc(lanes));
					at = __shfl_sync(0xffffffffu, at, 0) + __popc(lanes & ((1u << lane) - 1u));
					if (any) sm[a.o_task + at] = ((uint32_t)tb << 16) | ((uint32_t)g << 8) | (uint32_t)tx;
				}
			}
		} else {
			// every task; whole warps of columns where one or two are left over (+-16,
			// 32, 48, 64), those by one lane a candidate, below
			count = u.nb * a.tasks;
			for (int t = tid; t < count; t += nt) {
				const int b = a.div_tasks(t), v = t - b * a.tasks, g = a.div_cols(v);
				sm[a.o_task + t] = ((uint32_t)b << 16) | ((uint32_t)g << 8) | (uint32_t)(v - g * a.cols);
			}
		}
		if (hard) {  // uniform over the team
			// the window shifted by 1, 2, 3 bytes over the cells, copies 8 banks apart
			uint32_t* copies = sm + a.o_copy;
			for (int i = 4 * tid; i < a.wrows * SW; i += 4 * nt) {
				const uint4 x = *reinterpret_cast<const uint4*>(win + i);
				const uint32_t y = win[i + 4];
#pragma unroll
				for (int k = 1; k < 4; ++k)
					*reinterpret_cast<uint4*>(copies + (k - 1) * a.copy + i) =
						make_uint4(__funnelshift_r(x.x, x.y, 8 * k), __funnelshift_r(x.y, x.z, 8 * k),
					               __funnelshift_r(x.z, x.w, 8 * k), __funnelshift_r(x.w, y, 8 * k));
			}
			sync();
			if (count >= 0) {  // the columns left over
				const int left = nd - a.cols, more = u.nb * nd * left;
				for (int j0 = tid - lane; j0 < more; j0 += nt) {  // warp-uniform
					const int j = min(j0 + lane, more - 1), v = a.div_nd(j), b = left == 2 ? v >> 1 : v, iy = j - v * nd, ix = a.cols + v - b * left;
					const uint32_t* w = (ix & 3 ? copies + ((ix & 3) - 1) * a.copy : win) + iy * SW + ((16 * b + ix) >> 2);
					least_of(best, b, (exhaustive_rows<1, SW>(w, blkw + b * 64, 1) >> 5) << 15 | (uint32_t)(iy * nd + ix), lane);
				}
			}
			if (count < 0) exhaustive<GS, SW>(a, sm + a.o_task, n_tasks, win, copies, blkw, best, tid, nt);
			else if (a.rows == GA) exhaustive<GA, SW>(a, sm + a.o_task, count, win, copies, blkw, best, tid, nt);
			else exhaustive<GB, SW>(a, sm + a.o_task, count, win, copies, blkw, best, tid, nt);
		}
		sync();
		if (tid < u.nb) {
			const uint32_t key = best[tid];
			const int idx = (int)(key & 0x7fffu), iy = a.div_nd(idx);
			int32_t* o = a.out + 3 * (size_t)(u.blk0 + tid);
			o[0] = u.cy + iy - r;
			o[1] = u.cx + (idx - iy * nd) - r;
			o[2] = (int32_t)(key >> 15);
		}
		if (!LIST) break;  // a run per CTA
		sync();            // a list's next block overwrites the keys and the window
	}
}

template <class W, int MINB, int TEAMS>
umi_status launch(const ElimArgs& a, int threads, size_t smem, int sms, cudaStream_t st) {
	auto kern = full_me_elim_kernel<W, MINB, TEAMS>;
	UMI_TRY(umi::allow_shared(kern, smem));
	// a list's length is known on the GPU only: CTAs that fill it once take its blocks in turn
	const int grid = TEAMS ? std::min(a.units, MINB * sms) : a.units;
	kern<<<grid, threads, smem, st>>>(a);
	return umi::launch_status("full_me_elim_kernel");
}

}  // namespace

namespace umi {

// 16x16 argmin searches: any range 1..64, any width and alignment, lists and
// centres (full_me.cu says which come here).
umi_status full_me_elim(const uint8_t* cur, const uint8_t* ref, int h, int w, int r, const int32_t* centers,
                        int32_t* out, const int32_t* list, const int32_t* list_count, int max_slots, cudaStream_t st) {
	ElimArgs a{};
	a.cur = cur; a.ref = ref; a.centers = centers; a.out = out; a.list = list; a.list_count = list_count;
	a.h = h; a.w = w; a.r = r; a.nd = 2 * r + 1;
	a.nbx = w / 16;
	const int nby = h / 16, nblk = a.nbx * nby;
	a.slots = list ? std::min(max_slots, nblk) : nblk;
	if (a.slots <= 0) return UMI_OK;
	a.nchunk = ceil_div(a.nd, 2 * RC);
	const int per_b = a.nd * a.nchunk;
	int dev = 0, sms = 0;
	UMI_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
	UMI_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute"));
	a.nb = 1;
	if (!list && !centers) {
		// as many blocks per run as the threads and the cell rows hold, as long as the runs fill the GPU
		a.nb = std::max(1, std::min({MAXT / per_b, (Wide::QS - 3 - a.nd) / 16 + 1, MAXNB, a.nbx}));
		while (a.nb > 1 && ceil_div(a.nbx, a.nb) * nby < 2 * sms) --a.nb;
	}
	const bool narrow = a.nb == 1 && a.nd <= 65;
	const int SW = narrow ? Narrow::SW : Wide::SW, QS = narrow ? Narrow::QS : Wide::QS;
	a.runs_x = ceil_div(a.nbx, a.nb);
	a.units = list || centers ? a.slots : a.runs_x * nby;
	a.wrows = 2 * r + 16;
	a.wwords = ceil_div(16 * a.nb + 2 * r, 4);
	a.pieces = ceil_div(a.wwords, 4);
	a.qrows = 2 * r + 13;
	a.ncols = 16 * (a.nb - 1) + a.nd;
	a.spw = 32 / a.pieces;
	// Survivors cost three times a candidate of the exhaustive search, which takes
	// whole columns; below +-16 its copies of the window weigh more.  (Unrelated
	// frames, +-32, a limit of nd^2 / 8: 164 us, / 16 145, / 32 125, / 48 125.)
	a.limit = std::max(2 * a.nd, a.nd * a.nd / 32);
	a.cur_words = aligned(cur, 4) && w % 4 == 0;
	a.ref_pieces = aligned(ref, 16) && w % 16 == 0;
	a.div_x = Div::by(list || centers ? a.nbx : a.runs_x);
	a.mul16 = 16;
	a.mul64k = 1u << 16;
	a.cur_pieces = aligned(cur, 16) && w % 16 == 0;
	a.div_nd = SmallDiv::by(a.nd);
	a.div_task = SmallDiv::by(per_b);
	a.div_piece = SmallDiv::by(a.pieces);
	a.div_spw = SmallDiv::by(a.spw);
	// the exhaustive search of a run: rows per thread by the rows that a warp
	// works through, each task costing three halves of a row more
	a.cols = a.nd % 32 <= 2 && a.nd > 32 ? a.nd - a.nd % 32 : a.nd;
	const auto rows_cost = [&](int g) {
		return ceil_div(a.nb * a.cols * ceil_div(a.nd, g), narrow && !list ? 128 : 256) * (2 * g + 3);
	};
	a.rows = rows_cost(GB) < rows_cost(GA) ? GB : GA;
	a.tasks = a.cols * ceil_div(a.nd, a.rows);
	a.div_cols = SmallDiv::by(a.cols);
	a.div_tasks = SmallDiv::by(a.tasks);
	auto up4 = [](int n) { return (n + 3) & ~3; };
	const int threads = list ? 2 * (narrow ? Narrow::THREADS : Wide::THREADS)
	                         : narrow ? Narrow::THREADS : ceil_div(a.nb * per_b, 32) * 32;
	a.o_q = up4(a.wrows * SW + 4);
	// the exhaustive search's copies: 8, 16, 24 banks from the window; with fewer
	// rows than a thread takes it reads past a window's end
	a.copy = ceil_div(a.wrows * SW, 32) * 32 + 8;
	a.o_copy = ceil_div(a.o_q, 32) * 32 + 8;
	a.o_task = a.o_copy + 3 * a.copy + std::max(0, a.rows - a.nd) * SW;
	// a task in the rows of two of a column's threads may be listed twice
	a.o_blk = up4(std::max(a.o_q + (std::max(a.nd, RC) + 12) * QS,
	                       a.o_task + a.nb * a.nd * (ceil_div(a.nd, GS) + a.nchunk - 1)));
	a.o_cell = a.o_blk + 64 * a.nb;
	a.o_list = a.o_cell + 4 * a.nb;
	a.team_words = up4(a.o_list + a.nb * a.limit);
	const size_t smem = 4 * (size_t)a.team_words;
	if (list) {
		if (narrow) return launch<Narrow, 3, 2>(a, threads, 2 * smem, sms, st);
		return launch<Wide, 1, 2>(a, threads, 2 * smem, sms, st);
	}
	if (narrow) return launch<Narrow, 7, 0>(a, threads, smem, sms, st);
	if (smem > kSmemThree) return launch<Wide, 2, 0>(a, threads, smem, sms, st);
	return launch<Wide, 3, 0>(a, threads, smem, sms, st);
}

}  // namespace umi
