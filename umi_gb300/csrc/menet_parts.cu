// Data gradient of the 32 -> 32 channel 3x3 layers of the motion-proposal
// network (a convolution with transposed, flipped weights) on the tensor cores,
// at the accuracy of the FP32 pipe.
//
// The weights are bf16 values.  An fp32 gradient is the exact sum of three
// bf16 parts (8 + 8 + 8 mantissa bits, cut off, not rounded), so that all its
// products with a weight are exact and only their sums round.  The tensor
// core's fp32 sums truncate: the leading parts' products go to two
// accumulators, nine steps of 16 channels each, the others (2^-8 smaller) to a
// third, and the three are added with round to nearest.  The network's
// gradients are nearer to their 64-bit values than with the FP32 pipe here
// (medians of ten inputs: 2.7e-7 and 4.3e-7 at 720 x 1280, 3.3e-7 and 3.7e-7 at
// 256 x 1024).  The forward layers stay on the FP32 pipe: other roundings there
// move activations across the ReLU's zero, which changes gradients by 1e-5.
//
// Gradients between layers are kept twice: fp32 NCHW (weight gradient) and as
// parts, NHWC, 96 bf16 a pixel (32 channels of part 0, then of 1, 2).  Order of
// rows, strips and rolling accumulators are those of the inference layers
// (menet_rows_kernel in gemm_tc.cu): a CTA walks runs of rows y, y + d, ..., a
// strip (one row, 128 + 2 d pixels, here three boxes) is multiplied once by the
// stacked weights of every filter row that reads it.  Three rings of five
// 32-column accumulators fill 480 columns of TMEM.
//
// What bounds it: 18 MMAs of up to 96 columns a row of 128 pixels (about 40 ns
// each; 25 where the ring wraps) and, at 540 x 960, 330 MB of gradients and
// masks.  Layers at 4K (540 x 960): 62, 61 and 42 us (the last writes
// no parts) where the FP32 pipe took 230, 220 and 212, and 25 us once for the
// first parts; the whole pass 2151 -> 1687 us.
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "common.h"
#include "menet_roll.h"
#include "tc_common.cuh"

namespace umi {
void* tma_encode_fn();  // gemm_tc.cu
}

namespace {

using namespace umi_tc;

constexpr int CH = 32, PARTS = 3, PIXEL = CH * PARTS;  // bf16 values of a pixel
constexpr int BM = 128, MAXD = 8;
constexpr int SLOTS = 5, RINGS = 3, RING_COLS = SLOTS * 32;
constexpr int STAGES = 7;
constexpr uint32_t STRIP = ((BM + 2 * MAXD) * CH * 2 + 1023) & ~1023u;  // 9 216: one part of a strip
constexpr uint32_t STAGE = PARTS * STRIP, B_TILE = CH * CH * 2;         // 2 KB per tap
constexpr int EPI_WARPS = 8;  // two groups of four, taking alternate rows
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr size_t SMEM = (size_t)STAGES * STAGE + 9 * B_TILE + 1024 + 512;
static_assert(SMEM <= 227 * 1024 && RINGS * RING_COLS <= 512, "one CTA per SM");

struct PartsArgs {
	const float* mask;   // NCHW activations: zero where !(mask > 0)
	float* out;          // NCHW
	uint4* out_parts;    // or null
	int h, w, dil, xtiles;
	int* err;
	unsigned long long acc_wait_ns;  // limit of the epilogue's wait for a finished row (kWaitNs)
};

// a = p0 + p1 + p2 exactly, each the upper half of an fp32 word; an infinity is its own first part
__device__ __forceinline__ void split3(float a, uint32_t (&p)[PARTS]) {
	const uint32_t u = __float_as_uint(a);
	p[0] = u & 0xffff0000u;
	const float r = (u & 0x7fffffffu) == 0x7f800000u ? 0.0f : a - __uint_as_float(p[0]);
	p[1] = __float_as_uint(r) & 0xffff0000u;
	p[2] = __float_as_uint(r - __uint_as_float(p[1])) & 0xffff0000u;
}

// The pixel's 32 values as parts: six 32-byte stores.
__device__ __forceinline__ void store_parts(uint4* dst, const float (&v)[CH]) {
	uint32_t q[PARTS][CH / 2];
#pragma unroll
	for (int c = 0; c < CH; c += 2) {
		uint32_t a[PARTS], b[PARTS];
		split3(v[c], a);
		split3(v[c + 1], b);
#pragma unroll
		for (int k = 0; k < PARTS; ++k) q[k][c / 2] = __byte_perm(a[k], b[k], 0x7632);
	}
#pragma unroll
	for (int k = 0; k < PARTS; ++k)
#pragma unroll
		for (int i = 0; i < CH / 2; i += 8)
			asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + (k * CH / 2 + i) / 4),
			             "r"(q[k][i]), "r"(q[k][i + 1]), "r"(q[k][i + 2]), "r"(q[k][i + 3]), "r"(q[k][i + 4]), "r"(q[k][i + 5]),
			             "r"(q[k][i + 6]), "r"(q[k][i + 7])
			             : "memory");
}

__global__ void __launch_bounds__(256) to_parts_kernel(const float* __restrict__ in, uint4* __restrict__ parts, int P) {
	const int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= P) return;
	float v[CH];
#pragma unroll
	for (int c = 0; c < CH; ++c) v[c] = __ldg(in + (size_t)c * P + p);
	store_parts(parts + (size_t)p * (PIXEL * 2 / 16), v);
}

__global__ void __launch_bounds__(THREADS, 1)
	menet_dgrad_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const PartsArgs g,
	                   const int per) {
	extern __shared__ uint8_t smem_raw[];
	uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	uint8_t* bres = base + STAGES * STAGE;  // tap (dy, dx) at (3 dx + dy) * 2 KB: the dy of one dx adjacent
	uint64_t* full = reinterpret_cast<uint64_t*>(bres + 9 * B_TILE);
	uint64_t* empty = full + STAGES;
	uint64_t* accfull = empty + STAGES;    // [SLOTS]
	uint64_t* accempty = accfull + SLOTS;  // [SLOTS]
	uint64_t* drain = accempty + SLOTS;
	uint64_t* bready = drain + 1;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bready + 1);
	volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
	const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
	const int H = g.h, ntiles = g.xtiles * H, d = g.dil;
	const int t0 = blockIdx.x * per, t1 = min(ntiles, t0 + per);
	auto segment = [&](int s0, int& blk, int& y0, int& s1) {
		blk = s0 / H;
		int pend;
		umi_roll::row_of(H, d, s0 - blk * H, y0, pend);
		s1 = min(t1, blk * H + pend);
	};

	if (threadIdx.x == 0) {
		for (int s = 0; s < STAGES; ++s) {
			mbar_init(&full[s], 1);
			mbar_init(&empty[s], 1);
		}
		for (int a = 0; a < SLOTS; ++a) {
			mbar_init(&accfull[a], 1);
			mbar_init(&accempty[a], 4);
		}
		mbar_init(drain, 1);
		mbar_init(bready, 1);
		*abort_flag = 0;
		fence_mbar_init();
		tma_prefetch(&ta);
		tma_prefetch(&tb);
	}
	if (warp == 1) {
		tmem_alloc(tmem_slot, 512);
		tmem_relinquish();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = *tmem_slot;
	if (warp >= 2 && warp < 6) {  // one warp per lane quadrant clears every accumulator
#pragma unroll 1
		for (uint32_t c = 0; c < RINGS * RING_COLS; c += 32) tmem_zero32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c);
		tmem_wait_st();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();

	if (warp == 0 && lane == 0) {
		// ---- producer: weights once (tap ks = 3 dy + dx to slot 3 dx + dy), then every strip once
		int armed[STAGES];
		for (int s = 0; s < STAGES; ++s) armed[s] = -1;
		mbar_arrive_expect_tx(bready, 9 * B_TILE);
		for (int ks = 0; ks < 9; ++ks) tma_load_2d(bres + (3 * (ks % 3) + ks / 3) * B_TILE, &tb, bready, ks * CH, 0);
		const uint32_t sbytes = PARTS * (uint32_t)(BM + 2 * d) * CH * 2;
		uint32_t q = 0;
		bool go = true;
		for (int s0 = t0; go && s0 < t1 && !*abort_flag;) {
			int blk, y0, s1;
			segment(s0, blk, y0, s1);
			for (int i = 0; i < s1 - s0 + 2; ++i, ++q) {  // input row y0 + (i - 1) d
				const int s = (int)(q % STAGES);
				const uint32_t round = q / STAGES;
				if (!mbar_wait(&empty[s], (round & 1) ^ 1, abort_flag, g.err, kErrTimeoutEmpty)) { go = false; break; }
				mbar_arrive_expect_tx(&full[s], sbytes);
				armed[s] = (int)round;
				for (int k = 0; k < PARTS; ++k)
					tma_load_4d(base + s * STAGE + k * STRIP, &ta, &full[s], k * CH, blk * BM - d, y0 + (i - 1) * d, 0);
			}
			s0 = s1;
		}
		if (*abort_flag) {
			volatile int own = 0;
			for (int s = 0; s < STAGES; ++s)
				if (armed[s] >= 0) mbar_wait(&full[s], (uint32_t)armed[s] & 1, &own, g.err, kErrTimeoutFull);
			mbar_wait(bready, 0, &own, g.err, kErrTimeoutFull);
		}
	} else if (warp == 1) {
		// ---- MMA issuer: strip m of a run of `rows` output rows feeds rows
		// m - dy for dy in [lo, hi]; all lanes wait, one issues
		const uint32_t one = elect_one();
		bool ok = mbar_wait(bready, 0, abort_flag, g.err, kErrTimeoutFull);
		const uint64_t a_base = desc_kmajor_sw64(smem_u32(base)), b_base = desc_kmajor_sw64(smem_u32(bres));
		const uint32_t a_row = (uint32_t)(d * CH * 2) >> 4;
		uint32_t q = 0;  // strips so far
		int r0 = 0;      // output rows of the earlier runs
		for (int s0 = t0; ok && s0 < t1 && !*abort_flag;) {
			int blk, y0, s1;
			segment(s0, blk, y0, s1);
			const int rows = s1 - s0;
			for (int m = 0; m < rows + 2; ++m, ++q) {
				const umi_roll::Step st = umi_roll::step<SLOTS>(m, rows, r0);
				const int lo = st.lo, cnt = st.hi - st.lo + 1;
				if (lo == 0) {  // row r0 + m starts here: its accumulators must be drained and cleared
					const int r = r0 + m;
					if (!mbar_wait(&accempty[umi_roll::slot<SLOTS>(r)], ((uint32_t)(r / SLOTS) & 1) ^ 1, abort_flag, g.err,
					               kErrTimeoutAccEmpty)) {
						ok = false;
						break;
					}
					tc_fence_after();
				}
				const int s = (int)(q % STAGES);
				if (!mbar_wait(&full[s], (q / STAGES) & 1, abort_flag, g.err, kErrTimeoutFull)) {
					ok = false;
					break;
				}
				tc_fence_after();
				const int c1 = st.c1;  // blocks before the ring wraps to its first column
				const uint32_t id1 = idesc_f16(1u, BM, 32 * c1), id2 = idesc_f16(1u, BM, 32 * (cnt - c1));
				const uint64_t as = a_base + ((uint32_t)s * (STAGE >> 4));
#pragma unroll
				for (int k = 0; k < PARTS; ++k)
#pragma unroll
					for (int dx = 0; dx < 3; ++dx) {
						const uint64_t ad = as + (uint32_t)k * (STRIP >> 4) + (uint32_t)dx * a_row;
						const uint64_t bd = b_base + (uint32_t)(3 * dx + lo) * (B_TILE >> 4);
#pragma unroll
						for (int kk = 0; kk < CH / 16; ++kk) {
							const uint32_t ring = tmem + (uint32_t)((k ? 2 : kk) * RING_COLS);
							mma_f16(one, ring + 32u * (uint32_t)st.first, ad + 2 * kk, bd + 2 * kk, id1, true);
							if (c1 < cnt) mma_f16(one, ring, ad + 2 * kk, bd + (uint32_t)c1 * (B_TILE >> 4) + 2 * kk, id2, true);
						}
					}
				mma_commit(one, &empty[s]);  // the strip's only reader
				if (m >= 2) mma_commit(one, &accfull[umi_roll::slot<SLOTS>(r0 + m - 2)]);  // row m - 2 has all nine taps
			}
			r0 += rows;
			s0 = s1;
		}
		mma_commit(one, drain);
		volatile int own = 0;
		mbar_wait(drain, 0, &own, g.err, kErrTimeoutAccum);
	} else if (warp >= 2) {
		// ---- epilogue: group (w - 2) / 4 takes rows r = group mod 2; warp w
		// reads TMEM lanes 32 (w%4) .. +31 (pixels), clears the accumulators and
		// releases them before it stores
		const int qd = warp & 3, grp = (warp - 2) >> 2, P = g.h * g.w;
		for (int r = grp; t0 + r < t1; r += 2) {
			const int id = t0 + r, sl = umi_roll::slot<SLOTS>(r);
			__syncwarp();  // lanes without a pixel skip the stores below
			if (!mbar_wait_warp(&accfull[sl], (uint32_t)(r / SLOTS) & 1, abort_flag, g.err, kErrTimeoutAccum, g.acc_wait_ns))
				break;
			tc_fence_after();
			const uint32_t acc = tmem + ((uint32_t)(32 * qd) << 16) + 32u * (uint32_t)sl;
			float v[CH], t[CH];
			tmem_ld32(acc, v);
			tmem_ld32(acc + RING_COLS, t);
#pragma unroll
			for (int c = 0; c < CH; ++c) v[c] += t[c];
			tmem_ld32(acc + 2 * RING_COLS, t);
#pragma unroll
			for (int k = 0; k < RINGS; ++k) tmem_zero32(acc + k * RING_COLS);
			tmem_wait_st();
			tc_fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(&accempty[sl]);
			const int blk = id / H;
			int y, pend;
			umi_roll::row_of(H, d, id - blk * H, y, pend);
			const int x = blk * BM + 32 * qd + lane;
			if (x >= g.w) continue;
			const size_t p = (size_t)y * g.w + x;
#pragma unroll
			for (int c = 0; c < CH; ++c) {
				v[c] += t[c];
				if (!(__ldg(g.mask + (size_t)c * P + p) > 0.0f)) v[c] = 0.0f;
			}
			float* o = g.out + p;
#pragma unroll
			for (int c = 0; c < CH; ++c, o += P) *o = v[c];
			if (g.out_parts) store_parts(g.out_parts + p * (PIXEL * 2 / 16), v);
		}
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 1) {
		tc_fence_after();
		tmem_dealloc(tmem, 512);
	}
}

}  // namespace

namespace umi {

// NCHW (32, P) fp32 -> parts (P, 96) bf16.
umi_status menet_to_parts(const float* in, void* parts, int P, cudaStream_t st) {
	to_parts_kernel<<<ceil_div(P, 256), 256, 0, st>>>(in, static_cast<uint4*>(parts), P);
	return launch_status("to_parts_kernel");
}

// The 3x3 convolution of dilation dil of parts (h, w, 96) with wpack (32, 9*32)
// bf16 K-major (tap-major, then input channel), zero where !(mask > 0), to out
// (NCHW fp32) and out_parts (or null).  A wait that gives up leaves rows
// unwritten and its bit in *err; wait_ns: the epilogue's limit (0: kWaitNs).
umi_status menet_dgrad(const void* parts, const void* wpack, const float* mask, float* out, void* out_parts, int h, int w,
                       int dil, int* err, unsigned long long wait_ns, cudaStream_t st) {
	if (dil < 1 || dil > MAXD) return fail(UMI_ERR_UNSUPPORTED, "menet gradient: dilation %d", dil);
	auto enc = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(tma_encode_fn());
	if (!enc) return fail(UMI_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
	CUtensorMap ta, tb;
	{
		const cuuint64_t dims[4] = {PIXEL, (cuuint64_t)w, (cuuint64_t)h, 1};
		const cuuint64_t strides[3] = {PIXEL * 2, (cuuint64_t)w * PIXEL * 2, (cuuint64_t)h * w * PIXEL * 2};
		const cuuint32_t box[4] = {CH, (cuuint32_t)(BM + 2 * dil), 1, 1};
		const cuuint32_t es[4] = {1, 1, 1, 1};
		const CUresult rr = enc(&ta, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(parts), dims, strides, box, es,
		                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
		                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
		if (rr != CUDA_SUCCESS) return fail(UMI_ERR_CUDA, "menet gradient: activation tensor map (%d)", (int)rr);
	}
	{
		const cuuint64_t dims[2] = {9 * CH, CH};
		const cuuint64_t strides[1] = {9 * CH * 2};
		const cuuint32_t box[2] = {CH, CH};
		const cuuint32_t es[2] = {1, 1};
		const CUresult rr = enc(&tb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(wpack), dims, strides, box, es,
		                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
		                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
		if (rr != CUDA_SUCCESS) return fail(UMI_ERR_CUDA, "menet gradient: weight tensor map (%d)", (int)rr);
	}
	const PartsArgs g{mask, out, static_cast<uint4*>(out_parts), h, w, dil, ceil_div(w, BM), err,
	                  wait_ns ? wait_ns : kWaitNs};
	UMI_TRY(cuda_status(cudaFuncSetAttribute(menet_dgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM),
	                    "cudaFuncSetAttribute"));
	int dev = 0, sms = 0;
	UMI_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
	UMI_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute"));
	const int tiles = h * g.xtiles, per = ceil_div(tiles, std::min(tiles, sms));
	menet_dgrad_kernel<<<ceil_div(tiles, per), THREADS, SMEM, st>>>(ta, tb, g, per);
	return launch_status("menet_dgrad_kernel");
}

}  // namespace umi
