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
// summed.  On the benchmark's frame pairs that leaves about 30 of 4225 at
// +-32, on a panning camera 170; a block that keeps more than an eighth of
// its candidates (noise, unrelated frames) is searched exhaustively by the
// same CTA.
//
// What bounds it: the integer ALU pipe (the bound's `vabsdiff4`, the cells'
// byte permutations) and issue.  One CTA serves a run of NB horizontally
// adjacent blocks (their windows overlap, so the cells of the run's window are
// formed once), one block when the blocks come from a list or are moved by
// centres:
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
//      blocks with too many survivors: every candidate, thread = (column,
//      5 rows).
// Everything is shared memory and barriers: no workspace, no waits on other
// CTAs.
//
// Measured on a GB300, exhaustive search before -> now: 1080p +-32, blocks
// moved one by one 0.150 -> 0.0435 ms, panning camera 0.150 -> 0.064 ms; 1080p
// +-16 0.088 -> 0.025 ms; 4K +-64 2.19 -> 0.76 ms.  Content the bound does not
// serve pays for trying it: unrelated frames 0.150 -> 0.179 ms, independent
// noise 0.150 -> 0.218 ms.  62 % of the issue slots are used (27 warps per SM
// between barriers); by phase at 1080p +-32: pixels 12 us, cells 8, bound 14,
// survivors 5, exact sums 5.  Tried: two blocks per run on 160 threads (0.058
// ms), three on 224 (0.047), six cell rows per lane (0.048), a persistent form
// with the next run's pixels in flight (0.051), noise left to a second,
// warp-specialised launch (0.055 with noise at 0.173).
#include <algorithm>

#include "common.h"

namespace {

constexpr int RC = 33;       // candidate rows per pass of the bound, two passes per thread
constexpr int QS = 132;      // words per row of the cell words: columns of a run's window, a multiple of 4
constexpr int MAXT = 288;    // threads: the columns of one run
constexpr int MAXNB = 8;
constexpr int NC = MAXNB / 2;     // cells of a run per lane
constexpr size_t kSmemThree = 74 * 1024;  // dynamic shared memory that leaves room for three CTAs per SM
constexpr int CR = 3;        // cell rows per lane and step
constexpr int BG = 5;        // candidate rows per thread of the exhaustive search

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
	int wrows, wwords, sw;      // window: rows, words per row, row stride in words (an odd number of 16-byte pieces)
	int qrows, ncols, spw;      // cells: rows, columns; row pieces a warp forms at a time
	int pieces;                 // 16-byte pieces per window row
	int limit;                  // survivors a block may keep before it is searched exhaustively
	int cur_words;              // cur's rows are 4-byte aligned
	int ref_pieces;             // ref's rows are 16-byte aligned
	int cur_pieces;             // cur's rows are 16-byte aligned
	Div div_x;                  // by blocks or runs per block row
	SmallDiv div_nd, div_task, div_piece, div_spw;  // by nd, nd * nchunk, pieces, spw
	uint32_t mul16, mul64k;     // 16 and 2^16 (runtime values: the keys stay multiply-adds, off the ALU pipe)
	// shared memory offsets in words
	int copy, o_copy;           // stride and start of the shifted windows (over the cell words)
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

// SADs of BG candidate rows of one column against the block: the least, as
// sad * 16 + row.  p: the column's words, shifted so that they start on a word
// (row stride sw).  A ring of BG window rows meets each block row.
__device__ __forceinline__ uint32_t exhaustive_rows(const uint32_t* __restrict__ p, int sw,
                                                    const uint4* __restrict__ blk, int rows) {
	uint32_t ring[BG][4], acc[BG];
	auto fetch = [&](uint32_t (&v)[4]) {
#pragma unroll
		for (int k = 0; k < 4; ++k) v[k] = p[k];
		p += sw;
	};
#pragma unroll
	for (int q = 0; q < BG; ++q) acc[q] = 0;
#pragma unroll
	for (int q = 0; q < BG - 1; ++q) fetch(ring[q]);
#pragma unroll
	for (int py = 0; py < 16; ++py) {
		const uint4 c = blk[py];
		fetch(ring[(py + BG - 1) % BG]);
#pragma unroll
		for (int q = 0; q < BG; ++q) {
			const uint32_t(&v)[4] = ring[(py + q) % BG];
			acc[q] = sad4(c.x, v[0], acc[q]);
			acc[q] = sad4(c.y, v[1], acc[q]);
			acc[q] = sad4(c.z, v[2], acc[q]);
			acc[q] = sad4(c.w, v[3], acc[q]);
		}
	}
	uint32_t k = 0xffffffffu;
#pragma unroll
	for (int q = 0; q < BG; ++q)
		if (q < rows) k = min(k, acc[q] * 16u + (uint32_t)q);
	return k;
}

// Costs of rows y0 .. y0 + RC - 1 of one column (col: the shared address of
// cell row y0), packed: p[i] = cost[i] | cost[i + 16] << 16, p16 = cost[32].
// Returns the least cost * 64 + row (the first row among equals).
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
__device__ __forceinline__ Run run_of(const ElimArgs& a, int unit) {
	Run u{0, 0, 0, 1, 0, 0};
	if (a.list || a.centers) {
		u.blk0 = a.list ? a.list[unit] : unit;
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
__device__ __forceinline__ void load_run(const ElimArgs& a, const Run& u, uint32_t* win, uint32_t* blkw, int row0,
                                         int piece, int piece_rows, int tid, int nt) {
	const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
	const int gy0 = 16 * u.by + u.cy - a.r, gx0 = 16 * u.bx0 + u.cx - a.r;
	if (a.ref_pieces && (gx0 & 15) == 0 && gx0 >= 0 && gx0 + 16 * a.pieces <= a.w) {
		const uint8_t* src = a.ref + gx0 + 16 * piece;
		for (int row = row0; row < a.wrows; row += piece_rows)
			copy16(win + row * a.sw + 4 * piece, src + (size_t)min(max(gy0 + row, 0), a.h - 1) * a.w);
	} else {
		const size_t total = (size_t)a.h * a.w;
		for (int row = warp; row < a.wrows; row += nwarps) {
			const size_t off = (size_t)min(max(gy0 + row, 0), a.h - 1) * a.w;
			for (int k = lane; k < a.wwords; k += 32) {
				const int gx = gx0 + 4 * k;
				uint32_t* dst = win + row * a.sw + k;
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
__device__ __forceinline__ void form_cells(const ElimArgs& a, const uint32_t* __restrict__ win, uint32_t* __restrict__ q,
                                           int y0, int g, int cols, uint32_t lo, int sh) {
	const uint32_t lo2 = lo * 0x10001u, hi2 = lo2 + ((256u << sh) - 1u) * 0x10001u;
	const uint32_t* src = win + y0 * a.sw + 4 * g;
	uint32_t ring[3][8], sum[8];
	auto row = [&](uint32_t (&v)[8]) {
		const uint4 x = *reinterpret_cast<const uint4*>(src);
		src += a.sw;
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

// MINB: CTAs per SM (three at 72 registers; two where shared memory holds no
// more).  HALVES: a list of blocks with windows of more than 66 rows, whose
// length only the GPU knows.  One CTA per SM takes a block with all its threads
// if the list has no more blocks than there are CTAs, and otherwise works as two
// teams with a block each, of half the threads and shared memory, that never
// wait for one another.  (A fallback list of 130 blocks at 1080p, +-64, most of
// them hard: the pass around it 79 us with two CTAs per SM, 68 so; 28 000 blocks
// at 4K: the pass 1.17 ms with all threads on each block, 0.91 so.)
template <int MINB, bool HALVES>
__global__ void __launch_bounds__(HALVES ? 2 * MAXT : MAXT, MINB) full_me_elim_kernel(const ElimArgs a) {
	extern __shared__ __align__(16) uint32_t smem[];
	__shared__ uint32_t seeds[2][MAXNB], bests[2][MAXNB];
	__shared__ int cnts[2][MAXNB], totals[2];
	int units = a.units;
	if (a.list) units = min(units, *a.list_count);
	const bool teams = HALVES && units > (int)gridDim.x;
	const int team = teams ? (int)threadIdx.x / MAXT : 0, nteams = teams ? 2 : 1;
	const int tid = (int)threadIdx.x - team * MAXT, nt = teams ? MAXT : (int)blockDim.x;
	const int warp = tid >> 5, lane = tid & 31, nwarps = nt >> 5;
	auto sync = [&] {  // the threads of this team
		if (HALVES) asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(nt) : "memory");
		else __syncthreads();
	};
	uint32_t *seed = seeds[team], *best = bests[team];
	int *cnt = cnts[team], &total_cnt = totals[team];
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
		const Run u = run_of(a, unit);
		load_run(a, u, win, blkw, row0, piece, piece_rows, tid, nt);
		if (tid < MAXNB) {
			seed[tid] = 0xffffffffu;
			best[tid] = 0xffffffffu;
			cnt[tid] = 0;
		}
		if (tid == 0) total_cnt = 0;
		asm volatile("cp.async.wait_all;" ::: "memory");
		sync();
		// ---- 1. cells: cur's, by every warp for the scale; then the window's
		uint32_t sums[NC], mn = 0xffffffffu, mx = 0;
#pragma unroll
		for (int t = 0; t < NC; ++t) {
			if (32 * t >= 16 * u.nb) break;
			const int i = min(lane + 32 * t, 16 * u.nb - 1);
			const uint32_t* px = blkw + (i >> 4) * 64 + ((i >> 2) & 3) * 16 + (i & 3);
			uint32_t v = 0;
#pragma unroll
			for (int k = 0; k < 4; ++k) v = sad4(px[4 * k], 0u, v);
			sums[t] = v;
			mn = min(mn, v);
			mx = max(mx, v);
		}
		mn = __reduce_min_sync(0xffffffffu, mn);
		mx = __reduce_max_sync(0xffffffffu, mx);
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
			form_cells(a, win, q, (s0 + seg) * CR, min(gl, a.pieces - 1), gl < a.pieces ? a.ncols - 16 * gl : 0, lo, sh);
		sync();
		// ---- 2. bound
		const bool task = tb < u.nb;
		uint32_t p0[16], p1[16], l0 = 0, l1 = 0, k0 = 0xffffffffu, k1 = 0xffffffffu;
		if (task) {
			uint32_t c[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) c[i] = cell[4 * tb + i];
			const unsigned col = (unsigned)__cvta_generic_to_shared(q + 16 * tb + tx);
			k0 = bound_rows(col + 4u * QS * iy0, c, nd - iy0, a.mul16, a.mul64k, p0, l0);
			if (nd > RC) k1 = bound_rows(col + 4u * QS * iy1, c, RC, a.mul16, a.mul64k, p1, l1);
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
		uint32_t T = 0;
		for (int b = wb0; b <= min(wb1, u.nb - 1); ++b) {
			const uint32_t idx = seed[b] & 0x7fffu;
			const int iy = a.div_nd((int)idx), X = 16 * b + (int)idx - iy * nd + 8 * (lane & 1);
			const uint32_t* w = win + (iy + (lane >> 1)) * a.sw + (X >> 2);
			const uint32_t sel = 0x3210u + 0x1111u * (uint32_t)(X & 3);
			const uint2 c = *reinterpret_cast<const uint2*>(blkw + b * 64 + 2 * lane);
			const uint32_t w1 = w[1];
			const uint32_t s = sad4(c.x, __byte_perm(w[0], w1, sel), sad4(c.y, __byte_perm(w1, w[2], sel), 0u));
			const uint32_t U = __reduce_add_sync(0xffffffffu, s);
			if (lane == 0) atomicMin(&best[b], (U << 15) | idx);
			if (b == tb) T = min((U + (16u << sh) - 16u) >> sh, 4095u);
		}
		// ---- 4. survivors
		if (task && (min(k0, k1) >> 6) <= T) {
			uint32_t m0 = 0, m1 = 0;
			bool e0 = false, e1 = false;
			if ((k0 >> 6) <= T) {
				m0 = survivors(p0, T);
				if (nd < RC) m0 &= 0xffffffffu >> (32 - nd);
				e0 = nd >= RC && l0 <= T;
			}
			if ((k1 >> 6) <= T) {
				m1 = survivors(p1, T);
				e1 = l1 <= T;
			}
			const int n = __popc(m0) + __popc(m1) + e0 + e1;
			if (atomicAdd(&cnt[tb], n) + n <= a.limit) {
				uint32_t* dst = list + atomicAdd(&total_cnt, n);
				const uint32_t e = ((uint32_t)tb << 16) | (uint32_t)tx;
				if (e0) *dst++ = e + ((uint32_t)(iy0 + 32) << 8);
				if (e1) *dst++ = e + ((uint32_t)(iy1 + 32) << 8);
				for (; m0; m0 &= m0 - 1) *dst++ = e + ((uint32_t)(iy0 + __ffs((int)m0) - 1) << 8);
				for (; m1; m1 &= m1 - 1) *dst++ = e + ((uint32_t)(iy1 + __ffs((int)m1) - 1) << 8);
			}
		}
		sync();
		// ---- 5. exact sums
		int hard = 0;
		for (int b = 0; b < u.nb; ++b) hard |= (cnt[b] > a.limit) << b;
		const int n = hard == (1 << u.nb) - 1 ? 0 : total_cnt, sub = lane & 7;
		for (int j0 = 4 * warp; j0 < n; j0 += 4 * nwarps) {
			const uint32_t e = list[min(j0 + (lane >> 3), n - 1)];  // lanes past the end repeat the last candidate
			const int b = (int)(e >> 16), iy = (int)(e >> 8 & 255u), ix = (int)(e & 255u), X = 16 * b + ix;
			if (hard && __all_sync(0xffffffffu, hard >> b & 1)) continue;  // listed before its block had too many
			const uint32_t* w = win + (iy + sub) * a.sw + (X >> 2);
			const uint4* cr = reinterpret_cast<const uint4*>(blkw + b * 64) + sub;
			const uint32_t sel = 0x3210u + 0x1111u * (uint32_t)(X & 3);
			uint32_t s = 0;
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const uint4 c = cr[8 * h];
				uint32_t v[5];
#pragma unroll
				for (int k = 0; k < 5; ++k) v[k] = w[8 * h * a.sw + k];
				s = sad4(c.x, __byte_perm(v[0], v[1], sel), s);
				s = sad4(c.y, __byte_perm(v[1], v[2], sel), s);
				s = sad4(c.z, __byte_perm(v[2], v[3], sel), s);
				s = sad4(c.w, __byte_perm(v[3], v[4], sel), s);
			}
#pragma unroll
			for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
			if (sub == 0) atomicMin(&best[b], (s << 15) | (uint32_t)(iy * nd + ix));
		}
		if (hard) {  // uniform over the CTA
			// the window shifted by 1, 2, 3 bytes over the cells, copies 8 banks apart
			uint32_t* copies = sm + a.o_copy;
			for (int i = tid; i < a.wrows * a.sw; i += nt) {
				const uint32_t x = win[i], y = win[i + 1];
#pragma unroll
				for (int k = 1; k < 4; ++k) copies[(k - 1) * a.copy + i] = __funnelshift_r(x, y, 8 * k);
			}
			sync();
			const int ng = (nd + BG - 1) / BG, tasks = nd * ng, all = __popc(hard) * tasks;
			for (int t0 = tid - lane; t0 < all; t0 += nt) {  // warp-uniform
				const int t = min(t0 + lane, all - 1);       // lanes past the end repeat the last task
				const int hb = t / tasks, v = t - hb * tasks, g = a.div_nd(v), ix = v - g * nd;
				int m = hard;
				for (int k = 0; k < hb; ++k) m &= m - 1;
				const int b = __ffs(m) - 1;
				const uint32_t* w = (ix & 3 ? copies + ((ix & 3) - 1) * a.copy : win) + g * BG * a.sw + ((16 * b + ix) >> 2);
				const uint32_t e = exhaustive_rows(w, a.sw, reinterpret_cast<const uint4*>(blkw + b * 64), nd - g * BG);
				const uint32_t ekey = ((e >> 4) << 15) | (uint32_t)((g * BG + (int)(e & 15u)) * nd + ix);
				if (__all_sync(0xffffffffu, b == __shfl_sync(0xffffffffu, b, 0))) {
					const uint32_t least = __reduce_min_sync(0xffffffffu, ekey);
					if (lane == 0) atomicMin(&best[b], least);
				} else {
					atomicMin(&best[b], ekey);
				}
			}
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
		sync();  // a list's next block overwrites the keys and the window
	}
}

template <int MINB, bool HALVES>
umi_status launch(const ElimArgs& a, int threads, size_t smem, int sms, cudaStream_t st) {
	auto kern = full_me_elim_kernel<MINB, HALVES>;
	UMI_TRY(umi::allow_shared(kern, smem));
	// a list's length is known on the GPU only: CTAs that fill it once take its blocks in turn
	const int grid = a.list ? std::min(a.units, MINB * sms) : a.units;
	kern<<<grid, threads, smem, st>>>(a);
	return umi::launch_status("full_me_elim_kernel");
}

}  // namespace

namespace umi {

// Every 16x16 argmin search that full_me.cu does not serve from registers:
// any range 1..64, any width and alignment, lists and centres.
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
		a.nb = std::max(1, std::min({MAXT / per_b, (QS - 3 - a.nd) / 16 + 1, MAXNB, a.nbx}));
		while (a.nb > 1 && ceil_div(a.nbx, a.nb) * nby < 2 * sms) --a.nb;
	}
	a.runs_x = ceil_div(a.nbx, a.nb);
	a.units = list || centers ? a.slots : a.runs_x * nby;
	a.wrows = 2 * r + 16;
	a.wwords = ceil_div(16 * a.nb + 2 * r, 4);
	a.pieces = ceil_div(a.wwords, 4);
	a.sw = 4 * (a.pieces | 1);
	a.qrows = 2 * r + 13;
	a.ncols = 16 * (a.nb - 1) + a.nd;
	a.spw = 32 / a.pieces;
	a.limit = std::max(1, a.nd * a.nd / 8);
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
	auto up4 = [](int n) { return (n + 3) & ~3; };
	const bool halves = list && a.nd > 2 * RC;
	const int threads = halves ? 2 * MAXT : ceil_div(a.nb * per_b, 32) * 32;
	a.o_q = up4(a.wrows * a.sw + 4);
	// the exhaustive search's copies: 8, 16, 24 banks from the window; its last
	// row group reads up to BG - 1 rows past a window's end
	a.copy = ceil_div(a.wrows * a.sw, 32) * 32 + 8;
	a.o_copy = ceil_div(a.o_q, 32) * 32 + 8;
	a.o_blk = up4(std::max(a.o_q + (std::max(a.nd, RC) + 12) * QS, a.o_copy + 3 * a.copy + (BG - 1) * a.sw));
	a.o_cell = a.o_blk + 64 * a.nb;
	a.o_list = a.o_cell + 4 * a.nb;
	a.team_words = up4(a.o_list + a.nb * a.limit);
	const size_t smem = 4 * (size_t)a.team_words;
	if (halves) return launch<1, true>(a, threads, 2 * smem, sms, st);
	return smem > kSmemThree ? launch<2, false>(a, threads, smem, sms, st) : launch<3, false>(a, threads, smem, sms, st);
}

}  // namespace umi
