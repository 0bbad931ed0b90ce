// Integral image uint8 -> int32, sm_103a.
//
// Replaces the two Execute calls of main/iimg.cu:37-82 (a Loop-output prefix
// scan along x written transposed, applied twice) with one read of the uint8
// frame from HBM and one write of the int32 result.
//
// Two forms share this file.  umi_iimg_u8_i32 uses the band form (further
// down: column sums per group of bands, then one output pass).
// umi_iimg_u8_i32_noalloc keeps the tile form below, whose small tile sums
// fit the library's built-in scratch:
// the frame is cut into TH x TW tiles (64 x 256: a 1080p frame is 136 tiles,
// about one per SM).  With the inclusive integral image ii and a tile at
// (Y0, X0):
//   ii[y][x] = corner + sum_{X0<=x'<=x} top[x'] + sum_{Y0<=y'<=y} left[y'] + local[y][x]
//   top[x]   = sum over all rows above the tile of column x,
//   left[y]  = sum over all columns left of the tile of row y,
//   corner   = sum over the whole rectangle above-left of the tile,
//   local    = the 2-D prefix inside the tile.
// Kernel 1 (iimg_tile_sums) writes per-tile row sums, column sums and tile
// totals to a small workspace (about 3% of the output).  Kernel 2
// (iimg_tiles) loads its tile and computes the local prefix with warp-shuffle
// scans, then waits for kernel 1 (programmatic dependent launch: the wait is
// griddepcontrol.wait, so everything before it overlaps kernel 1), adds the
// carries (at most nty + ntx + nty*ntx small-array reads per tile, issued as
// independent loads) and writes the tile with 16-byte stores.
#include <cuda.h>

#include <mutex>

#include "common.h"

namespace {

constexpr int NT = 256;         // threads: 8 warps
constexpr int NW = NT / 32;
constexpr int RPW = 8;          // rows per warp
constexpr int TH = NW * RPW;    // 64 tile rows
constexpr int CPL = 8;          // columns per lane
constexpr int TW = 32 * CPL;    // 256 tile columns
constexpr int MAXNTY = 64;      // carries unrolled up to this many tile rows (frames up to 4096 rows)

struct IimgGeom {
	int h, w, ntx, nty;
	int vec_in;   // in is 8-byte aligned and w % 8 == 0
	int vec_out;  // out is 16-byte aligned and w % 4 == 0
	int32_t* rowsum;   // [h][ntx]
	int32_t* colsum;   // [nty][w]
	int32_t* tilesum;  // [nty][ntx]
};

__device__ __forceinline__ void pdl_wait() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
	asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}
__device__ __forceinline__ void pdl_trigger() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
	asm volatile("griddepcontrol.launch_dependents;");
#endif
}

// The lane's 8 pixels of row y starting at column x, zeros past the edges.
__device__ __forceinline__ uint2 load8(const uint8_t* __restrict__ in, const IimgGeom& g, int y, int x) {
	if (y >= g.h) return make_uint2(0, 0);
	const uint8_t* row = in + (size_t)y * g.w;
	if (g.vec_in && x + 7 < g.w) return __ldg(reinterpret_cast<const uint2*>(row + x));
	uint32_t lo = 0, hi = 0;
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		if (x + k < g.w) lo |= (uint32_t)__ldg(row + x + k) << (8 * k);
		if (x + 4 + k < g.w) hi |= (uint32_t)__ldg(row + x + 4 + k) << (8 * k);
	}
	return make_uint2(lo, hi);
}

__device__ __forceinline__ void unpack8(uint2 p, uint32_t v[8]) {
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		v[k] = (p.x >> (8 * k)) & 0xffu;
		v[4 + k] = (p.y >> (8 * k)) & 0xffu;
	}
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
		if (lane >= o) v += n;
	}
	return v;
}

__global__ void __launch_bounds__(NT) iimg_tile_sums(const uint8_t* __restrict__ in, const IimgGeom g) {
	__shared__ uint32_t colpart[NW][TW];
	__shared__ uint32_t warptot[NW];
	pdl_wait();  // when launched after an earlier kernel that may write `in`
	pdl_trigger();
	const int tx = blockIdx.x, ty = blockIdx.y;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int X0 = tx * TW, Y0 = ty * TH;
	const int y0 = Y0 + warp * RPW, x = X0 + CPL * lane;
	uint2 raw[RPW];
#pragma unroll
	for (int r = 0; r < RPW; ++r) raw[r] = load8(in, g, y0 + r, x);
	uint32_t col[CPL] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
	for (int r = 0; r < RPW; ++r) {
		uint32_t v[CPL];
		unpack8(raw[r], v);
		uint32_t s = 0;
#pragma unroll
		for (int k = 0; k < CPL; ++k) { s += v[k]; col[k] += v[k]; }
		s = __reduce_add_sync(0xffffffffu, s);
		if (lane == 0 && y0 + r < g.h) g.rowsum[(size_t)(y0 + r) * g.ntx + tx] = (int32_t)s;
	}
#pragma unroll
	for (int k = 0; k < CPL; ++k) colpart[warp][CPL * lane + k] = col[k];
	__syncthreads();
	{
		const int c = threadIdx.x;  // NT == TW: one column per thread
		uint32_t s = 0;
#pragma unroll
		for (int i = 0; i < NW; ++i) s += colpart[i][c];
		if (X0 + c < g.w) g.colsum[(size_t)ty * g.w + X0 + c] = (int32_t)s;
		s = __reduce_add_sync(0xffffffffu, s);
		if (lane == 0) warptot[warp] = s;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t t = 0;
#pragma unroll
		for (int i = 0; i < NW; ++i) t += warptot[i];
		g.tilesum[(size_t)ty * g.ntx + tx] = (int32_t)t;
	}
}

__global__ void __launch_bounds__(NT) iimg_tiles(const uint8_t* __restrict__ in, int32_t* __restrict__ out,
                                                 const IimgGeom g) {
	__shared__ uint32_t wtot[NW][TW];  // per-warp column totals, then their exclusive prefix over warps
	__shared__ uint32_t topw[NW];      // per-warp totals of the top-carry x-scan
	__shared__ uint32_t lefty[TH];     // inclusive y-prefix of the left carries
	__shared__ uint32_t cornerp[NW];
	const int tx = blockIdx.x, ty = blockIdx.y;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int X0 = tx * TW, Y0 = ty * TH;
	const int y0 = Y0 + warp * RPW, x = X0 + CPL * lane;

	// Local 2-D prefix.  The input is not written by kernel 1, so it is read
	// before the dependency wait and overlaps kernel 1.
	uint2 raw[RPW];
#pragma unroll
	for (int r = 0; r < RPW; ++r) raw[r] = load8(in, g, y0 + r, x);
	uint32_t loc[RPW][CPL];
	uint32_t col[CPL] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
	for (int r = 0; r < RPW; ++r) {
		uint32_t v[CPL];
		unpack8(raw[r], v);
#pragma unroll
		for (int k = 1; k < CPL; ++k) v[k] += v[k - 1];
		const uint32_t excl = warp_incl_scan(v[CPL - 1], lane) - v[CPL - 1];
#pragma unroll
		for (int k = 0; k < CPL; ++k) {
			col[k] += v[k] + excl;
			loc[r][k] = col[k];
		}
	}
#pragma unroll
	for (int k = 0; k < CPL; ++k) wtot[warp][CPL * lane + k] = col[k];
	__syncthreads();
	{
		const int c = threadIdx.x;
		uint32_t run = 0;
#pragma unroll
		for (int i = 0; i < NW; ++i) {
			const uint32_t t = wtot[i][c];
			wtot[i][c] = run;
			run += t;
		}
	}

	// Carries from kernel 1.
	pdl_wait();
	pdl_trigger();
	uint32_t topc;  // inclusive x-prefix (within this warp's 32 columns) of the top carries
	{
		const int c = threadIdx.x, xc = X0 + c;
		uint32_t s = 0;
		if (xc < g.w) {
#pragma unroll
			for (int t = 0; t < MAXNTY; ++t)
				if (t < ty) s += (uint32_t)__ldcg(g.colsum + (size_t)t * g.w + xc);
		}
		topc = warp_incl_scan(s, lane);
		if (lane == 31) topw[warp] = topc;
	}
	if (threadIdx.x < TH) {
		const int y = Y0 + threadIdx.x;
		uint32_t s = 0;
		if (y < g.h) {
#pragma unroll 8
			for (int t = 0; t < tx; ++t) s += (uint32_t)__ldcg(g.rowsum + (size_t)y * g.ntx + t);
		}
		// rows are spread over warps 0 and 1: scan within each, stitch below
		lefty[threadIdx.x] = warp_incl_scan(s, lane);
	}
	{
		uint32_t s = 0;
		const int n = ty * tx;
		for (int i = threadIdx.x; i < n; i += NT) {
			const int a = i / tx, b = i - a * tx;
			s += (uint32_t)__ldcg(g.tilesum + (size_t)a * g.ntx + b);
		}
		s = __reduce_add_sync(0xffffffffu, s);
		if (lane == 0) cornerp[warp] = s;
	}
	__syncthreads();
	uint32_t corner = 0;
#pragma unroll
	for (int i = 0; i < NW; ++i) corner += cornerp[i];
	// Top carry prefix for this lane's 8 columns: the warp-level scans of
	// columns [32*wv, 32*wv+32) are in topc of warp wv; columns of this lane
	// are CPL*lane .. CPL*lane+7, owned by warp (CPL*lane)/32.
	__shared__ uint32_t topx[TW];
	topx[threadIdx.x] = topc;
	__syncthreads();
	uint32_t topv[CPL];
#pragma unroll
	for (int k = 0; k < CPL; ++k) {
		const int c = CPL * lane + k;
		uint32_t t = topx[c];
		const int seg = c >> 5;
		for (int sgi = 0; sgi < seg; ++sgi) t += topw[sgi];
		topv[k] = t + corner + wtot[warp][c];
	}
	uint32_t lbase = 0;
	if (warp * RPW >= 32) lbase = lefty[31];  // rows 32..63: add the total of rows 0..31
#pragma unroll
	for (int r = 0; r < RPW; ++r) {
		const int y = y0 + r;
		if (y >= g.h) break;
		const uint32_t lv = lefty[warp * RPW + r] + lbase;
		int32_t o[CPL];
#pragma unroll
		for (int k = 0; k < CPL; ++k) o[k] = (int32_t)(loc[r][k] + topv[k] + lv);
		int32_t* dst = out + (size_t)y * g.w + x;
		if (g.vec_out && x + 7 < g.w) {
			reinterpret_cast<int4*>(dst)[0] = make_int4(o[0], o[1], o[2], o[3]);
			reinterpret_cast<int4*>(dst)[1] = make_int4(o[4], o[5], o[6], o[7]);
		} else {
#pragma unroll
			for (int k = 0; k < CPL; ++k)
				if (x + k < g.w) dst[k] = o[k];
		}
	}
}

size_t ws_bytes(int h, int w) {
	const size_t ntx = umi::ceil_div(w, TW), nty = umi::ceil_div(h, TH);
	auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
	return al((size_t)h * ntx * 4) + al(nty * (size_t)w * 4) + al(nty * ntx * 4);
}

// ---------------------------------------------------------------------------
// Band form (umi_iimg_u8_i32).  The frame is cut into bands of RB rows over
// the full width and the bands into groups of GB bands (128 rows).  With
// V[b][x] = sum of column x over all rows above band b,
//   ii[y][x] = sum_{x'<=x} V[b][x'] + sum_{band rows y'<=y} sum_{x'<=x} in[y'][x'],
//   V[b][x]  = sum_{groups g' above the group of b} S[g'][x] + W[b][x],
// where S[g][x] is the column sum of group g and W[b][x] the column sum of the
// bands of its group above b.  Kernel 1 (one CTA per group and chunk of 128
// columns) reads every group once and writes W and S (uint16: at most 128 *
// 255), the row sums of its chunk and the totals of W and S over it.  Kernel 2
// (one CTA per band and segment of 1024 columns) loads its pixels, waits for
// kernel 1 (programmatic dependent launch: its launch and pixel loads overlap
// kernel 1), takes what lies left of its segment from the chunks' row sums and
// totals (a few values per thread), forms V from at most ceil(h / 128)
// independent loads per column, scans its RB rows and its V row along x with
// one block-wide scan of RB + 1 values per thread, and writes its rows with
// 32-byte stores.  Two launches, both parallel over the whole frame; no
// grid-wide wait.  Before, one CTA walked a whole band: 270
// CTAs with two dependent steps each at 4K.  Measured (graph replay, us,
// before -> now): 2160 x 3840 22.5 -> 17.2, 1440 x 2560 16.1 -> 9.7, 1081 x
// 1923 (no aligned row) 16.5 -> 9.0, 1080 x 1920 6.9 -> 6.6.  32-byte stores
// give 1 us of that at 4K (16-byte ones touch every sector twice).  Frames of
// at most 2048 columns are one segment of 256 threads: two of 128 cost more
// in the sums to the left than they gain (1080p 7.3).
constexpr int RB = 8;          // rows per band
constexpr int GB = 16;         // bands per group
constexpr int GCT = 16;        // kernel-1 threads across the columns of a group (x CPL = 128 columns)
constexpr int CHUNK = GCT * CPL;   // columns of a kernel-1 CTA
static_assert(GB * GCT == NT, "kernel 1: one thread per band and 8 columns");

struct BandGeom {
	int h, w, nb, ng, wpad, nch;
	int vec_in, vec_out;
	int vec_out8;    // rows of out are 32-byte aligned
	int left;        // a CTA per segment, several per band: kernel 1 writes the last three arrays
	uint16_t* wsum;  // [ng * GB][wpad]  W
	uint16_t* gsum;  // [ng][wpad]       S
	uint16_t* rsum;  // [nch][ng * GB * RB]  row sums per chunk
	uint32_t* wtot;  // [nch][ng * GB]   W summed over the chunk
	uint32_t* gtot;  // [nch][ng]        S summed over the chunk
};

// Frames up to this width are one segment of 256 threads.
constexpr int kOneSegment = 256 * CPL;

// Workspace layout: offsets of the arrays above, the bytes up to the last one and
// those of the first two alone, which serve any frame.
struct BandWork {
	size_t off[5], bytes, least;
	BandWork(int h, int w) {
		const size_t nb = umi::ceil_div(h, RB), ng = umi::ceil_div(nb, (size_t)GB);
		const size_t wpad = (size_t)umi::ceil_div(w, CPL) * CPL, nch = umi::ceil_div(w, CHUNK);
		const size_t n[5] = {ng * GB * wpad * 2, ng * wpad * 2, nch * ng * GB * RB * 2, nch * ng * GB * 4, nch * ng * 4};
		bytes = 0;
		for (int i = 0; i < 5; ++i) {
			off[i] = bytes;
			bytes += (n[i] + 255) & ~size_t(255);
		}
		least = off[2];
		if (w <= kOneSegment) bytes = least;
	}
};

// Rows y0 .. y0 + RB - 1 of a thread's 8 columns.  Rows of any alignment are
// read as three aligned words each, decided once for all of them (a decision
// per row keeps the loads from being issued together), where every word lies
// in the frame.
__device__ __forceinline__ void load_rows(const uint8_t* __restrict__ in, const IimgGeom& g, int y0, int x,
                                          uint2 (&raw)[RB]) {
	const size_t o = (size_t)y0 * g.w + x;
	if (!g.vec_in && x + 7 < g.w && y0 + RB <= g.h && o >= 3 && o + (size_t)(RB - 1) * g.w + 12 <= (size_t)g.h * g.w) {
		uint32_t w[RB][3];
#pragma unroll
		for (int r = 0; r < RB; ++r) {
			const uint32_t* s = reinterpret_cast<const uint32_t*>((reinterpret_cast<uintptr_t>(in) + o + (size_t)r * g.w) &
			                                                      ~(uintptr_t)3);
#pragma unroll
			for (int k = 0; k < 3; ++k) w[r][k] = __ldg(s + k);
		}
#pragma unroll
		for (int r = 0; r < RB; ++r) {
			const int sh = 8 * (int)((reinterpret_cast<uintptr_t>(in) + o + (size_t)r * g.w) & 3);
			raw[r] = make_uint2(__funnelshift_r(w[r][0], w[r][1], sh), __funnelshift_r(w[r][1], w[r][2], sh));
		}
	} else {
#pragma unroll
		for (int r = 0; r < RB; ++r) raw[r] = load8(in, g, y0 + r, x);
	}
}

__global__ void __launch_bounds__(NT) iimg_group_sums(const uint8_t* __restrict__ in, const BandGeom g) {
	__shared__ __align__(16) uint32_t cs[GB][CHUNK];
	__shared__ uint32_t btot[GB];  // total of each band
	pdl_trigger();
	const int gi = blockIdx.y, j = threadIdx.x / GCT, c = threadIdx.x % GCT;
	const int xs = blockIdx.x * CHUNK, x0 = xs + c * CPL;
	IimgGeom ig{};
	ig.h = g.h; ig.w = g.w; ig.vec_in = g.vec_in;
	uint32_t s[CPL] = {};
	uint32_t rows[RB / 2] = {};  // row sums of these 8 columns, two rows per word (at most 128 * 255 per chunk)
	if (x0 < g.w) {
		const int y0 = (gi * GB + j) * RB;
		uint2 raw[RB];
		load_rows(in, ig, y0, x0, raw);
#pragma unroll
		for (int r = 0; r < RB; ++r) {
			uint32_t v[CPL];
			unpack8(raw[r], v);
			uint32_t t = 0;
#pragma unroll
			for (int k = 0; k < CPL; ++k) {
				s[k] += v[k];
				t += v[k];
			}
			rows[r >> 1] += t << (16 * (r & 1));
		}
	}
	if (g.left) {
#pragma unroll
		for (int i = 0; i < RB / 2; ++i)
#pragma unroll
			for (int o = 1; o < GCT; o <<= 1) rows[i] += __shfl_xor_sync(0xffffffffu, rows[i], o);
	}
	if (g.left && c == 0) {
		static_assert(RB == 8, "one 16-byte store per band");
		*reinterpret_cast<uint4*>(g.rsum + ((size_t)blockIdx.x * g.ng * GB + gi * GB + j) * RB) =
			make_uint4(rows[0], rows[1], rows[2], rows[3]);
		uint32_t t = 0;
#pragma unroll
		for (int i = 0; i < RB / 2; ++i) t += (rows[i] & 0xffffu) + (rows[i] >> 16);
		btot[j] = t;
	}
	*reinterpret_cast<uint4*>(&cs[j][c * CPL]) = make_uint4(s[0], s[1], s[2], s[3]);
	*reinterpret_cast<uint4*>(&cs[j][c * CPL + 4]) = make_uint4(s[4], s[5], s[6], s[7]);
	__syncthreads();
	if (g.left && threadIdx.x < GB) {
		uint32_t run = 0;
		for (int k = 0; k < (int)threadIdx.x; ++k) run += btot[k];
		g.wtot[(size_t)blockIdx.x * g.ng * GB + gi * GB + threadIdx.x] = run;
		if (threadIdx.x == GB - 1) g.gtot[(size_t)blockIdx.x * g.ng + gi] = run + btot[GB - 1];
	}
	if (threadIdx.x < CHUNK) {  // one column per thread: exclusive prefix over the group's bands
		const int x = xs + threadIdx.x;
		if (x < g.w) {
			uint32_t run = 0;
#pragma unroll
			for (int k = 0; k < GB; ++k) {
				g.wsum[(size_t)(gi * GB + k) * g.wpad + x] = (uint16_t)run;
				run += cs[k][threadIdx.x];
			}
			g.gsum[(size_t)gi * g.wpad + x] = (uint16_t)run;
		}
	}
}

__device__ __forceinline__ void add_u16x8(uint32_t (&v)[CPL], uint4 p) {
	v[0] += p.x & 0xffffu; v[1] += p.x >> 16;
	v[2] += p.y & 0xffffu; v[3] += p.y >> 16;
	v[4] += p.z & 0xffffu; v[5] += p.z >> 16;
	v[6] += p.w & 0xffffu; v[7] += p.w >> 16;
}

// NT2: threads, 8 columns each.  WALK: a CTA takes a band's segments one after the
// other, its sums carried along (a workspace without the sums per chunk).
template <int NT2, bool WALK>
__global__ void __launch_bounds__(NT2, NT2 == 128 ? 6 : 2) iimg_band_out(const uint8_t* __restrict__ in, int32_t* __restrict__ out,
                                                      const BandGeom g) {
	constexpr int NW2 = NT2 / 32, SEG = NT2 * CPL;
	static_assert(SEG % CHUNK == 0, "segments start on chunks");
	__shared__ uint32_t wtot[NW2][RB + 1];
	__shared__ uint32_t left[NW2][RB + 1];  // per warp: sums over the chunks left of the segment (rows, then the V row)
	__shared__ __align__(16) uint32_t rowbuf[NW2][4][32 * CPL];
	const int b = blockIdx.x, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
	const int y0 = b * RB;
	IimgGeom ig{};
	ig.h = g.h; ig.w = g.w; ig.vec_in = g.vec_in;
	uint32_t carry[RB + 1] = {};  // WALK: of each row and of the V row, left of the segment
	int seg = WALK ? 0 : blockIdx.y;
	do {
		const int x0 = seg * SEG + threadIdx.x * CPL;
		const bool live = x0 < g.w;
		uint2 raw[RB] = {};
		if (live) load_rows(in, ig, y0, x0, raw);
		pdl_wait();
		const int gb = b / GB, nleft = WALK ? 0 : seg * (SEG / CHUNK);  // groups above, chunks to the left
		uint32_t vv[CPL] = {};
		if (live) {  // V = W of this band + S of every group above
			add_u16x8(vv, __ldcg(reinterpret_cast<const uint4*>(g.wsum + (size_t)b * g.wpad + x0)));
#pragma unroll 8
			for (int q = 0; q < gb; ++q) add_u16x8(vv, __ldcg(reinterpret_cast<const uint4*>(g.gsum + (size_t)q * g.wpad + x0)));
		}
		if (nleft) {
			uint32_t rl[CPL] = {}, vl = 0;
			for (int c = threadIdx.x; c < nleft; c += NT2) {
				add_u16x8(rl, __ldcg(reinterpret_cast<const uint4*>(g.rsum + ((size_t)c * g.ng * GB + b) * RB)));
				vl += __ldcg(g.wtot + (size_t)c * g.ng * GB + b);
			}
			for (int c = wp; c < nleft; c += NW2)
				for (int q = lane; q < gb; q += 32) vl += __ldcg(g.gtot + (size_t)c * g.ng + q);
#pragma unroll
			for (int r = 0; r < RB; ++r) rl[r] = __reduce_add_sync(0xffffffffu, rl[r]);
			vl = __reduce_add_sync(0xffffffffu, vl);
			if (lane == 0) {
#pragma unroll
				for (int r = 0; r < RB; ++r) left[wp][r] = rl[r];
				left[wp][RB] = vl;
			}
		}
		// thread totals of each row and of the V row, scanned over the block
		uint32_t tsum[RB + 1];
#pragma unroll
		for (int r = 0; r < RB; ++r) {
			uint32_t v[CPL];
			unpack8(raw[r], v);
			uint32_t t = 0;
#pragma unroll
			for (int k = 0; k < CPL; ++k) t += v[k];
			tsum[r] = t;
		}
		{
			uint32_t t = 0;
#pragma unroll
			for (int k = 0; k < CPL; ++k) t += vv[k];
			tsum[RB] = t;
		}
		uint32_t ex[RB + 1];
#pragma unroll
		for (int r = 0; r <= RB; ++r) {
			const uint32_t inc = warp_incl_scan(tsum[r], lane);
			ex[r] = inc - tsum[r];
			if (lane == 31) wtot[wp][r] = inc;
		}
		__syncthreads();
#pragma unroll
		for (int r = 0; r <= RB; ++r) {
#pragma unroll
			for (int k = 0; k < NW2 - 1; ++k) ex[r] += k < wp ? wtot[k][r] : 0u;
			if (nleft)
#pragma unroll
				for (int k = 0; k < NW2; ++k) ex[r] += left[k][r];
			if constexpr (WALK) {
				ex[r] += carry[r];
#pragma unroll
				for (int k = 0; k < NW2; ++k) carry[r] += wtot[k][r];
			}
		}
		// outputs: T(x) = V-row prefix, plus the running column sum of the row prefixes
		uint32_t T[CPL];
		{
			uint32_t tp = ex[RB];
#pragma unroll
			for (int k = 0; k < CPL; ++k) {
				tp += vv[k];
				T[k] = tp;
			}
		}
#pragma unroll
		for (int r = 0; r < RB; ++r) {
			uint32_t rp = ex[r];
#pragma unroll
			for (int k = 0; k < CPL; ++k) {
				rp += (k < 4 ? (raw[r].x >> (8 * k)) : (raw[r].y >> (8 * (k - 4)))) & 0xffu;
				T[k] += rp;
			}
			const int y = y0 + r;
			if (y >= g.h) break;
			int32_t* op = out + (size_t)y * g.w + x0;
			if (g.vec_out8) {  // w % 8 == 0: every live thread has 8 columns
				if (live)
					asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(op), "r"(T[0]), "r"(T[1]),
					             "r"(T[2]), "r"(T[3]), "r"(T[4]), "r"(T[5]), "r"(T[6]), "r"(T[7])
					             : "memory");
			} else if (g.vec_out) {  // w % 4 == 0
				if (live) reinterpret_cast<int4*>(op)[0] = make_int4(T[0], T[1], T[2], T[3]);
				if (x0 + 7 < g.w) reinterpret_cast<int4*>(op)[1] = make_int4(T[4], T[5], T[6], T[7]);
			} else {  // any alignment: the warp's 256 columns through shared memory, four rows at a time
				uint32_t* row = rowbuf[wp][r & 3];
				*reinterpret_cast<uint4*>(row + CPL * lane) = make_uint4(T[0], T[1], T[2], T[3]);
				*reinterpret_cast<uint4*>(row + CPL * lane + 4) = make_uint4(T[4], T[5], T[6], T[7]);
				if ((r & 3) == 3 || y == g.h - 1) {
					__syncwarp();
					const int xw = x0 - CPL * lane + lane;
					for (int i = 0; i <= (r & 3); ++i) {
						int32_t* o = out + (size_t)(y - (r & 3) + i) * g.w + xw;
#pragma unroll
						for (int k = 0; k < CPL; ++k)  // 128 contiguous bytes per store
							if (xw + 32 * k < g.w) o[32 * k] = (int32_t)rowbuf[wp][i][32 * k + lane];
					}
					__syncwarp();
				}
			}
		}
		if constexpr (WALK) __syncthreads();  // the next segment's totals overwrite these
	} while (WALK && ++seg * SEG < g.w);
}

cudaLaunchAttribute pdl_attr() {
	cudaLaunchAttribute a;
	a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	a.val.programmaticStreamSerializationAllowed = 1;
	return a;
}

}  // namespace

extern "C" size_t umi_iimg_u8_i32_workspace_bytes(int32_t h, int32_t w) {
	if (h <= 0 || w <= 0) return 0;
	return BandWork(h, w).bytes;
}

extern "C" umi_status umi_iimg_u8_i32(const uint8_t* in, int32_t* out, int32_t h, int32_t w, void* workspace,
                                      size_t workspace_bytes, void* stream) {
	if (h < 0 || w < 0) return umi::fail(UMI_ERR_INVALID_ARG, "iimg: negative size %dx%d", h, w);
	if (h == 0 || w == 0) return umi::ok();
	if (!in || !out || !workspace) return umi::fail(UMI_ERR_INVALID_ARG, "iimg: null pointer");
	if (!umi::aligned(workspace, 16)) return umi::fail(UMI_ERR_INVALID_ARG, "iimg: workspace not 16-byte aligned");
	const BandWork work(h, w);
	if (workspace_bytes < work.least)
		return umi::fail(UMI_ERR_NO_MEMORY, "iimg: workspace of %zu bytes, need %zu", workspace_bytes, work.bytes);
	if ((int64_t)h * w > ((int64_t)1 << 31) / 255)
		return umi::fail(UMI_ERR_UNSUPPORTED, "iimg: %dx%d frame: sums could exceed int32", h, w);
	BandGeom g{};
	g.h = h; g.w = w;
	g.nb = umi::ceil_div(h, RB);
	g.ng = umi::ceil_div(g.nb, GB);
	g.wpad = umi::ceil_div(w, CPL) * CPL;
	g.nch = umi::ceil_div(w, CHUNK);
	g.vec_in = umi::aligned(in, 8) && (w % 8) == 0;
	g.vec_out = umi::aligned(out, 16) && (w % 4) == 0;
	g.vec_out8 = umi::aligned(out, 32) && (w % 8) == 0;
	// a frame of at most 2048 columns is one segment (nothing lies left of it); a
	// wider one has a CTA per segment where the workspace holds the sums to the
	// left of them, else one per band (graph replays, us: 1440 x 2560 9.3 and 11.3,
	// 1081 x 2561 10.8 and 13.1, 2160 x 3840 15.5 and 14.5)
	const bool segments = w > kOneSegment && workspace_bytes >= work.bytes;
	const int nt2 = segments ? 128 : 256;
	g.left = segments;
	char* ws = static_cast<char*>(workspace);
	g.wsum = reinterpret_cast<uint16_t*>(ws + work.off[0]);
	g.gsum = reinterpret_cast<uint16_t*>(ws + work.off[1]);
	g.rsum = reinterpret_cast<uint16_t*>(ws + work.off[2]);
	g.wtot = reinterpret_cast<uint32_t*>(ws + work.off[3]);
	g.gtot = reinterpret_cast<uint32_t*>(ws + work.off[4]);
	const cudaStream_t st = umi::as_stream(stream);
	// kernel 1 follows whatever the stream ran before: plain launch
	iimg_group_sums<<<dim3(g.nch, g.ng), NT, 0, st>>>(in, g);
	UMI_TRY(umi::launch_status("iimg_group_sums"));
	cudaLaunchAttribute attr[1] = {pdl_attr()};
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(g.nb, segments ? umi::ceil_div(w, nt2 * CPL) : 1);
	cfg.blockDim = dim3(nt2);
	cfg.stream = st;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	auto kern = segments ? iimg_band_out<128, false> : w <= kOneSegment ? iimg_band_out<256, false> : iimg_band_out<256, true>;
	UMI_TRY(umi::cuda_status(cudaLaunchKernelEx(&cfg, kern, in, out, g), "iimg_band_out"));
	return umi::ok();
}

// ---------------------------------------------------------------------------
// Allocation-free integral image.
//
// Some callers of this library cannot allocate device memory at all: a plugin
// inside a host application that owns the GPU memory budget, code that runs
// where cudaMalloc is not allowed (a real-time loop with a no-allocation
// rule, a host callback), or a caller that simply has no allocator to hand a
// workspace from.  umi_iimg_u8_i32_noalloc serves them: the tile sums go to
// a scratch array compiled into this library, so the caller passes only the
// frame and the output.
//
// The scratch is a file-scope __device__ array of kNoAllocScratchBytes
// (1 MiB: the tile sums of every frame the int32 limit accepts, up to 4096
// rows; the largest accepted frame has h*w*255 < 2^31, about 8.42 Mpx, so
// 3840x2160 is served and 4096x2160 is refused by that limit); every GPU that
// loads the library holds it until the process exits.  Host code cannot use
// the array's name as a device address, so the first call in each CUDA
// context (with that context current) looks the address up with
// cudaGetSymbolAddress and caches it under the context handle; make that
// first call before any stream capture.  A context destroyed and re-created
// while the library stays loaded (cudaDeviceReset) can come back with the
// same handle: such a caller calls umi_iimg_noalloc_forget() after the reset.
// All calls share the one array: calls that overlap on the GPU (different
// streams, different host threads) race on it and must be serialised by the
// caller.  Nothing in the scratch needs to start at zero: kernel 1 writes
// every entry kernel 2 reads.
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(1) << 20;
static_assert(kNoAllocScratchBytes == UMI_IIMG_NOALLOC_SCRATCH_BYTES, "header and library disagree");
static __device__ __align__(256) unsigned char g_iimg_scratch[kNoAllocScratchBytes];

// Scratch address per CUDA context (the module, and so the array, is loaded
// once per context: the primary context of each device, or a context the
// caller made current through the driver API).
constexpr int kMaxContexts = 64;
std::mutex g_scratch_mu;
struct ScratchEntry { void* ctx; void* addr; };
ScratchEntry g_scratch[kMaxContexts] = {};
int g_scratch_n = 0;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
CtxGetCurrentFn ctx_get_current_fn() {
	static CtxGetCurrentFn fn = nullptr;
	static std::once_flag once;
	std::call_once(once, [] {
		cudaDriverEntryPointQueryResult q;
		void* p = nullptr;
		if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
		    q == cudaDriverEntryPointSuccess)
			fn = reinterpret_cast<CtxGetCurrentFn>(p);
	});
	return fn;
}

umi_status scratch_address(void** out) {
	int dev = 0;
	UMI_TRY(umi::cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
	// the runtime makes the device's primary context current if none is yet
	UMI_TRY(umi::cuda_status(cudaFree(nullptr), "cudaFree(0) (context initialisation)"));
	auto get = ctx_get_current_fn();
	if (!get) return umi::fail(UMI_ERR_CUDA, "iimg_noalloc: cuCtxGetCurrent unavailable");
	CUcontext ctx = nullptr;
	if (get(&ctx) != CUDA_SUCCESS || !ctx) return umi::fail(UMI_ERR_CUDA, "iimg_noalloc: no current CUDA context");
	std::lock_guard<std::mutex> lock(g_scratch_mu);
	for (int i = 0; i < g_scratch_n; ++i)
		if (g_scratch[i].ctx == ctx) {
			*out = g_scratch[i].addr;
			return UMI_OK;
		}
	if (g_scratch_n == kMaxContexts) return umi::fail(UMI_ERR_UNSUPPORTED, "iimg_noalloc: more than %d contexts", kMaxContexts);
	void* p = nullptr;
	UMI_TRY(umi::cuda_status(cudaGetSymbolAddress(&p, g_iimg_scratch), "cudaGetSymbolAddress"));
	g_scratch[g_scratch_n++] = {reinterpret_cast<void*>(ctx), p};
	*out = p;
	return UMI_OK;
}

}  // namespace

extern "C" umi_status umi_iimg_u8_i32_noalloc(const uint8_t* in, int32_t* out, int32_t h, int32_t w, void* stream) {
	if (h < 0 || w < 0) return umi::fail(UMI_ERR_INVALID_ARG, "iimg_noalloc: negative size %dx%d", h, w);
	if (h == 0 || w == 0) return umi::ok();
	if (!in || !out) return umi::fail(UMI_ERR_INVALID_ARG, "iimg_noalloc: null pointer");
	if (ws_bytes(h, w) > kNoAllocScratchBytes)
		return umi::fail(UMI_ERR_NO_MEMORY, "iimg_noalloc: a %dx%d frame needs %zu scratch bytes, the built-in scratch holds %zu",
		                 h, w, ws_bytes(h, w), kNoAllocScratchBytes);
	if (umi::ceil_div(h, TH) > MAXNTY)
		return umi::fail(UMI_ERR_UNSUPPORTED, "iimg_noalloc: %d rows (max %d)", h, MAXNTY * TH);
	if ((int64_t)h * w > ((int64_t)1 << 31) / 255)
		return umi::fail(UMI_ERR_UNSUPPORTED, "iimg_noalloc: %dx%d frame: sums could exceed int32", h, w);
	void* scratch = nullptr;
	UMI_TRY(scratch_address(&scratch));
	IimgGeom g{};
	g.h = h; g.w = w;
	g.ntx = umi::ceil_div(w, TW);
	g.nty = umi::ceil_div(h, TH);
	g.vec_in = umi::aligned(in, 8) && (w % 8) == 0;
	g.vec_out = umi::aligned(out, 16) && (w % 4) == 0;
	auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
	char* ws = static_cast<char*>(scratch);
	g.rowsum = reinterpret_cast<int32_t*>(ws);
	g.colsum = reinterpret_cast<int32_t*>(ws + al((size_t)h * g.ntx * 4));
	g.tilesum = reinterpret_cast<int32_t*>(ws + al((size_t)h * g.ntx * 4) + al((size_t)g.nty * w * 4));
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(g.ntx, g.nty);
	cfg.blockDim = dim3(NT);
	cfg.stream = umi::as_stream(stream);
	cudaLaunchAttribute attr[1] = {pdl_attr()};
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	UMI_TRY(umi::cuda_status(cudaLaunchKernelEx(&cfg, iimg_tile_sums, in, g), "iimg_tile_sums"));
	UMI_TRY(umi::cuda_status(cudaLaunchKernelEx(&cfg, iimg_tiles, in, out, g), "iimg_tiles"));
	return umi::ok();
}

extern "C" void umi_iimg_noalloc_forget(void) {
	std::lock_guard<std::mutex> lock(g_scratch_mu);
	g_scratch_n = 0;
}
