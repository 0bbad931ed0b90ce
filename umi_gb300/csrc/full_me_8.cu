// Full search of 8x8 blocks (argmin) over uint8 frames, sm_103a: every block
// of the frame at its own place, any range 1..64, any width and alignment.
// Lists and centres stay with the general kernel of full_me.cu, whose result
// this one reproduces: the smallest SAD, the first displacement in raster
// order among equals, reference pixels clamped to the frame.
//
// What bounds it: the packed-SAD instruction (vabsdiff4 ... add, four pixels,
// half rate): a block's (2r+1)^2 x 16 of them.  The split keeps everything
// else off that pipe and out of shared memory:
//  * a CTA takes a strip of up to 32 horizontally adjacent blocks and stages
//    their common window once (neighbours share most of it);
//  * a lane is one block, a warp takes four neighbouring horizontal
//    displacements at a time: they share the three words that a row's eight
//    pixels can touch, and their byte shifts are constants;
//  * the block's 16 words stay in registers while the window's rows stream by;
//    a row serves the eight vertical displacements it can belong to, whose sums
//    are a ring of eight registers, so one 64-bit and one 32-bit load feed 64
//    packed SADs;
//  * the window is kept twice, the second copy one word further on, so that the
//    64-bit loads are aligned for every group of displacements.
// Three CTAs of nine warps fit an SM with 72 registers a thread (27.5 us with
// 96 and two CTAs).  Measured, and before with one window per block and four
// shifted copies of it: 717 x 1278 +-16 23.3 us, before 98.5; 1080 x 1920 +-7
// 24.5 and 95.0, +-32 183 and 372.  The packed SADs alone would take 12.3 us of
// the 23.3: the rest is byte shifts, keys, and staging that the other CTAs hide
// only in part.
#include <algorithm>

#include "common.h"

namespace {

constexpr int kLanes = 32;      // blocks per strip
constexpr int kMaxWarps = 9;    // +-16: eight groups of four displacements and the last one

struct Args8 {
	const uint8_t *cur, *ref;
	int32_t* out;
	int h, w, r, ndx;
	int nbx, nb, runs_x;  // blocks per row, per strip; strips per row
	int lanes;            // lanes a warp gives to the blocks of a strip: a power of two >= nb
	int units;            // groups of four horizontal displacements
	int groups, chunks;   // groups of eight window rows (after the first) per chunk of vertical displacements; chunks
	int wrows, wwords;    // window rows and words staged
	int pitch;            // words from row to row, even
};

__device__ __forceinline__ uint32_t sad4(uint32_t a, uint32_t b, uint32_t c) {
	uint32_t d;
	asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
	return d;
}

// Pixels gx .. gx + 3 of the row at byte offset `off`, columns clamped: two
// aligned words where all four and the words' other bytes are the frame's.
__device__ __forceinline__ uint32_t pixels(const uint8_t* f, size_t total, size_t off, int gx, int w) {
	const size_t o = off + gx;
	if (gx >= 0 && gx + 4 <= w && o >= 4 && o + 8 <= total) {
		const uintptr_t p = reinterpret_cast<uintptr_t>(f) + o;
		const uint32_t* s = reinterpret_cast<const uint32_t*>(p & ~(uintptr_t)3);
		return __funnelshift_r(__ldg(s), __ldg(s + 1), 8 * (int)(p & 3));
	}
	uint32_t v = 0;
#pragma unroll
	for (int k = 0; k < 4; ++k) v |= (uint32_t)__ldg(f + off + min(max(gx + k, 0), w - 1)) << (8 * k);
	return v;
}

// Eight window rows (KIND 0 a chunk's first ones, 2 its last ones) against the
// block rows they can meet.  At row j of the eight, block row py belongs to the
// vertical displacement whose sum is in slot (j - py) & 7; it starts at py = 0
// and is complete after py = 7, as displacement iy + j of the search.  off[s]
// is the horizontal displacement, or beyond every key where there is none.
template <int NIX, int KIND>
__device__ __forceinline__ void rows8(const uint32_t* __restrict__ wp, int pitch, const uint32_t (&c)[8][2],
                                      uint32_t (&acc)[NIX][8], uint32_t& key, int iy, int ndx,
                                      const uint32_t (&off)[NIX]) {
#pragma unroll
	for (int j = 0; j < 8; ++j) {
		const uint2 w01 = *reinterpret_cast<const uint2*>(wp + j * pitch);
		const uint32_t w2 = NIX > 1 ? wp[j * pitch + 2] : 0;
#pragma unroll
		for (int s = 0; s < NIX; ++s) {
			const uint32_t a = s ? __funnelshift_r(w01.x, w01.y, 8 * s) : w01.x;
			const uint32_t b = s ? __funnelshift_r(w01.y, w2, 8 * s) : w01.y;
#pragma unroll
			for (int py = KIND == 2 ? j : 0; py <= (KIND == 0 ? j : 7); ++py) {
				uint32_t& sum = acc[s][(j - py) & 7];
				sum = sad4(c[py][1], b, sad4(c[py][0], a, py ? sum : 0u));
			}
		}
		if ((KIND != 0 || j == 7) && iy + j < ndx) {
			const uint32_t first = (uint32_t)((iy + j) * ndx);
#pragma unroll
			for (int s = 0; s < NIX; ++s) key = min(key, (acc[s][(j + 1) & 7] << 15) + (first + off[s]));
		}
	}
}

// Vertical displacements iy .. iy + 8 groups, horizontal ones 4 u .. 4 u + 3.
template <int NIX>
__device__ __forceinline__ uint32_t unit8(const Args8& a, const uint32_t* wp, const uint32_t (&c)[8][2], int u, int iy) {
	uint32_t acc[NIX][8], off[NIX];
#pragma unroll
	for (int s = 0; s < NIX; ++s) off[s] = 4 * u + s < a.ndx ? 4 * u + s : 0x40000000u;  // sums are below 2^14
	uint32_t key = 0xffffffffu;
	const int step = 8 * a.pitch;
	rows8<NIX, 0>(wp, a.pitch, c, acc, key, iy - 7, a.ndx, off);
	wp += step;
	++iy;
#pragma unroll 1
	for (int g = 1; g < a.groups; ++g, wp += step, iy += 8) rows8<NIX, 1>(wp, a.pitch, c, acc, key, iy, a.ndx, off);
	rows8<NIX, 2>(wp, a.pitch, c, acc, key, iy, a.ndx, off);
	return key;
}

// SPLIT: a warp holds several groups of displacements of fewer blocks.
template <bool SPLIT>
__global__ void __launch_bounds__(32 * kMaxWarps, 3) full_me_8_kernel(const Args8 a) {
	extern __shared__ __align__(16) uint32_t sm[];
	__shared__ __align__(16) uint32_t blk[8][2 * kLanes];
	__shared__ uint32_t best[kLanes];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
	const int by = blockIdx.x / a.runs_x, bx0 = (blockIdx.x - by * a.runs_x) * a.nb;
	const int count = min(a.nb, a.nbx - bx0);
	const int gy0 = 8 * by - a.r, gx0 = 8 * bx0 - a.r;
	const size_t total = (size_t)a.h * a.w;
	uint32_t* win1 = sm + a.wrows * a.pitch;  // word k holds word k + 1 of the window's row
	if (threadIdx.x < kLanes) best[threadIdx.x] = 0xffffffffu;
	for (int k = lane; k < a.wwords; k += 32) {
#pragma unroll 4
		for (int row = warp; row < a.wrows; row += nwarps) {
			const uint32_t v = pixels(a.ref, total, (size_t)min(max(gy0 + row, 0), a.h - 1) * a.w, gx0 + 4 * k, a.w);
			sm[row * a.pitch + k] = v;
			if (k) win1[row * a.pitch + k - 1] = v;
		}
	}
	for (int i = threadIdx.x; i < 8 * 2 * count; i += blockDim.x) {
		const int row = i / (2 * count), k = i - row * 2 * count;
		blk[row][k] = pixels(a.cur, total, (size_t)(8 * by + row) * a.w, 8 * bx0 + 4 * k, a.w);
	}
	__syncthreads();
	const int sub = SPLIT ? lane / a.lanes : 0, l = min(SPLIT ? lane - sub * a.lanes : lane, count - 1);
	uint32_t c[8][2];
#pragma unroll
	for (int py = 0; py < 8; ++py) {
		const uint2 v = *reinterpret_cast<const uint2*>(&blk[py][2 * l]);
		c[py][0] = v.x;
		c[py][1] = v.y;
	}
	uint32_t key = 0xffffffffu;
	if (SPLIT) {
		const int slots = a.units * a.chunks, per_warp = 32 / a.lanes;
		for (int first = warp * per_warp; first < slots; first += nwarps * per_warp) {
			const int slot = min(first + sub, slots - 1), chunk = slot / a.units, u = slot - chunk * a.units;
			const int iy = 8 * a.groups * chunk;
			key = min(key, unit8<4>(a, ((u & 1) ? win1 : sm) + iy * a.pitch + 2 * l + (u & ~1), c, u, iy));
		}
	} else {
		for (int u = warp; u < a.units; u += nwarps) {
			const uint32_t* wp = ((u & 1) ? win1 : sm) + 2 * l + (u & ~1);
			key = min(key, 4 * u + 1 == a.ndx ? unit8<1>(a, wp, c, u, 0) : unit8<4>(a, wp, c, u, 0));
		}
	}
	atomicMin(&best[l], key);
	__syncthreads();
	if (threadIdx.x < count) {
		const uint32_t k = best[threadIdx.x];
		const int idx = (int)(k & 0x7fffu), iy = idx / a.ndx;
		int32_t* o = a.out + 3 * ((size_t)by * a.nbx + bx0 + threadIdx.x);
		o[0] = iy - a.r;
		o[1] = idx - iy * a.ndx - a.r;
		o[2] = (int32_t)(k >> 15);
	}
}

}  // namespace

namespace umi {

umi_status full_me_8(const uint8_t* cur, const uint8_t* ref, int h, int w, int r, int32_t* out, cudaStream_t st) {
	Args8 a{};
	a.cur = cur; a.ref = ref; a.out = out;
	a.h = h; a.w = w; a.r = r;
	a.ndx = 2 * r + 1;
	a.nbx = w / 8;
	a.units = ceil_div(a.ndx, 4);
	const int nby = h / 8, all = ceil_div(2 * r, 8);
	int dev = 0, sms = 0;
	UMI_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
	UMI_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute"));
	// The split, by its clocks on the busiest SM: a chunk of `groups` costs a
	// warp 64 groups + 8 (row, block row) pairs of eight packed SADs, two clocks
	// each, an SM runs four warps at once; staging costs about a fifth of a clock
	// a word.  Whole strips of 32 blocks with one chunk have no masked lanes and
	// no rows in two chunks, but a small frame has too
	// few of them (240 x 320 +-16: 6.4 us, whole strips 10.8; +-32 14.1 and 28.6).
	int64_t best = INT64_MAX;
	for (int lanes = kLanes; lanes >= 1; lanes /= 2)
		for (int groups = all; groups >= 1; groups = groups > 1 ? ceil_div(groups, 2) : 0) {
			const bool split = lanes < kLanes;
			if (!split && groups < all) continue;
			const int runs = ceil_div(a.nbx, lanes), nb = ceil_div(a.nbx, runs), chunks = ceil_div(all, groups);
			const int64_t per_sm = ceil_div((int64_t)runs * nby, (int64_t)sms);
			const int64_t warps = ceil_div((int64_t)a.units * chunks * lanes, (int64_t)32);
			const int64_t unit = 16 * (64 * groups + 8) * (split ? 9 : 8) / 8;
			const int64_t words = (int64_t)8 * (chunks * groups + 1) * (2 * nb + a.units);
			const int64_t cost = std::max<int64_t>(ceil_div(warps, (int64_t)kMaxWarps) * 4, per_sm * warps) * unit / 4 +
			                     per_sm * words / 5;
			if (cost < best) {
				best = cost;
				a.lanes = lanes;
				a.groups = groups;
			}
		}
	a.runs_x = ceil_div(a.nbx, a.lanes);
	a.nb = ceil_div(a.nbx, a.runs_x);
	a.runs_x = ceil_div(a.nbx, a.nb);
	a.chunks = ceil_div(all, a.groups);
	a.wrows = 8 * (a.chunks * a.groups + 1);
	a.wwords = 2 * a.nb + a.units;
	a.pitch = (a.wwords + 1) & ~1;
	// one round of a warp's groups where they fit, else rounds of eight; four
	// warps at least, for the staging
	const int rounds = ceil_div(a.units * a.chunks * a.lanes, 32);
	const int warps = rounds <= kMaxWarps ? std::max(rounds, 4) : 8;
	const size_t smem = 2 * (size_t)a.wrows * a.pitch * sizeof(uint32_t);
	auto kern = a.lanes < kLanes ? full_me_8_kernel<true> : full_me_8_kernel<false>;
	UMI_TRY(allow_shared(kern, smem));
	kern<<<a.runs_x * nby, 32 * warps, smem, st>>>(a);
	return launch_status("full_me_8_kernel");
}

}  // namespace umi
