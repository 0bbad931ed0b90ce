// Learned motion proposal for block motion estimation (sm_103a).
//
// No counterpart in the reference: a small CNN proposes one motion vector
// per 16x16 block from the 1/4-downsampled frame pair, the UMI SAD kernel
// (full_me.cu) refines it in a small window, and blocks whose refined SAD is
// above a threshold fall back to exhaustive search.
//
// Network (all hand-written kernels below; fp32 master parameters, bf16
// weights in the forward/backward arithmetic, fp32 accumulation):
//   x0  = ((cur, ref) box-averaged 4x4 - 128) / 32                  (2, H4, W4)
//   a_l = ReLU(conv3x3_dil(a_{l-1}; W_l, b_l)), dilations 1, 2, 4, 8 (32, H4, W4)
//   mv  = Wh . a4[:, 4 cells x 4 cells of the block] + bh          (nblk, 2)
// The dilations give a receptive field of +-15 cells (+-60 pixels at full
// resolution).  mv is in units of 16 pixels.  Training minimises the smooth-L1
// distance to full-search vectors / 16 with Adam.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "common.h"
#include "me_pipeline.h"
#include "menet_train.cuh"

namespace umi {
umi_status menet_conv_tc(const void* in, void* out, const void* wpack, const float* bias, int h, int w, int dil,
                         int* err, cudaStream_t st);
// The layers' data gradient on the tensor cores at fp32 accuracy (menet_parts.cu).
umi_status menet_to_parts(const float* in, void* parts, int P, cudaStream_t st);
umi_status menet_dgrad(const void* parts, const void* wpack, const float* mask, float* out, void* out_parts, int h, int w,
                       int dil, int* err, unsigned long long wait_ns, cudaStream_t st);
}

namespace {

constexpr int CH = 32;       // channels of every hidden layer
constexpr int NL = 4;        // conv layers
constexpr int HEADF = CH * 16;  // head features per block (32 channels x 4 x 4 cells)
constexpr int DIL[NL] = {1, 2, 4, 8};
constexpr int CIN[NL] = {2, CH, CH, CH};
constexpr int NT = 256;

// ---- parameter layout (fp32 master copy; bf16 copies are derived from it)
struct Layout {
	int w[NL], b[NL], wh, bh, total;
	Layout() {
		int o = 0;
		for (int l = 0; l < NL; ++l) {
			w[l] = o; o += CH * CIN[l] * 9;
			b[l] = o; o += CH;
		}
		wh = o; o += 2 * HEADF;
		bh = o; o += 2;
		total = o;
	}
};

// ---- workspace layout for a frame of h x w pixels, in `have` bytes.  What a
// backward pass takes over from the forward pass and what the motion search
// needs lie apart; the rest is scratch that the passes share.  A workspace
// smaller than `bytes` (at least `least`) holds fewer rows of partial sums, and
// one too small for every layer's forward weights at once takes them in turn.
struct Work {
	int H4, W4, P, nbx, nby, nblk;
	size_t x0, act[NL], wt[NL], pred, centers, list, count, alist, amv, err;
	size_t wf[NL];           // forward: weights (menet_train.cuh), fp32, after the first layer every value twice
	size_t nhwc[2], wtc[NL]; // tensor-core inference: bf16 (H4, W4, 32) activations, packed weights
	size_t slot[3], part;    // backward: gradients, fp32 or as bf16 parts (menet_parts.cu); partial sums
	int htx, htiles, units;  // the head's tiles; rows of 32 columns that the weight gradients walk
	int parts, head_parts;   // rows of partial sums
	bool whole;              // every layer's forward weights at once
	size_t least, bytes;
	Work(int h, int w, size_t have = ~(size_t)0) {
		H4 = h / 4; W4 = w / 4; P = H4 * W4;
		nbx = w / 16; nby = h / 16; nblk = nbx * nby;
		htx = umi::ceil_div(nbx, 8); htiles = htx * nby;
		units = umi::ceil_div(W4, 32) * H4;
		auto al = [](size_t n) { return (n + 255) & ~size_t(255); };
		size_t o = 0;
		auto take = [&](size_t n) { size_t r = o; o += al(n); return r; };
		x0 = take(sizeof(float) * 2 * P);
		for (int l = 0; l < NL; ++l) act[l] = take(sizeof(float) * CH * P);
		for (int l = 0; l < NL; ++l) wt[l] = l ? take(2 * CH * CIN[l] * 9) : 0;  // bf16, for the data gradient
		pred = take(sizeof(float) * 2 * nblk);
		centers = take(sizeof(int32_t) * 2 * nblk);
		list = take(sizeof(int32_t) * nblk);
		count = take(sizeof(int32_t) * 4);  // [0] fallback blocks, [2] audited blocks
		alist = take(sizeof(int32_t) * nblk);
		amv = take(sizeof(int32_t) * 3 * nblk);
		err = take(sizeof(int32_t));
		const size_t scratch = o;
		constexpr size_t ROW = sizeof(float) * (CH * CH * 9 + CH), HEAD_ROW = sizeof(float) * (2 * HEADF + 3);
		constexpr size_t WF0 = sizeof(float) * CH * CIN[0] * 9, WF = sizeof(float) * 2 * CH * CH * 9;
		for (int i = 0; i < 2; ++i) nhwc[i] = take((size_t)P * 64);
		for (int l = 1; l < NL; ++l) wtc[l] = take(2 * CH * 9 * CH);
		const size_t infer = o;
		o = scratch;
		for (int i = 0; i < 3; ++i) slot[i] = take((size_t)P * 3 * CH * 2);
		part = o;
		parts = std::min(units, menet_train::PARTS);
		head_parts = std::min(htiles, menet_train::HEAD_PARTS);
		const size_t forward = scratch + al(WF0) + (NL - 1) * al(WF);
		bytes = std::max({infer, forward, part + al(std::max(parts * ROW, head_parts * HEAD_ROW))});
		least = std::max({infer, scratch + al(WF0) + al(WF), part + al(std::max(ROW, HEAD_ROW))});
		const size_t end = std::min(have, bytes);
		const size_t room = end > part ? end - part : 0;
		parts = (int)std::min<size_t>(parts, room / ROW);
		head_parts = (int)std::min<size_t>(head_parts, room / HEAD_ROW);
		whole = end >= forward;
		wf[0] = scratch;
		for (int l = 1; l < NL; ++l) wf[l] = scratch + al(WF0) + (whole ? l - 1 : 0) * al(WF);
	}
	template <class T> T* at(void* ws, size_t off) const { return reinterpret_cast<T*>(static_cast<char*>(ws) + off); }
};

// ------------------------------------------------------------------ kernels
__global__ void downsample4_kernel(const uint8_t* __restrict__ cur, const uint8_t* __restrict__ ref,
                                   float* __restrict__ x0, int w, int H4, int W4) {
	const int P = H4 * W4;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * P; i += gridDim.x * blockDim.x) {
		const int c = i / P, p = i - c * P, y = p / W4, x = p - y * W4;
		const uint8_t* src = (c == 0 ? cur : ref) + (size_t)(4 * y) * w + 4 * x;
		int s = 0;
#pragma unroll
		for (int dy = 0; dy < 4; ++dy)
#pragma unroll
			for (int dx = 0; dx < 4; ++dx) s += src[(size_t)dy * w + dx];
		x0[i] = (float)s * (1.0f / 512.0f) - 4.0f;  // (box mean - 128) / 32, exact in fp32
	}
}

// Adam (Kingma & Ba, 2015) on the fp32 master parameters.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const float gi = g[i];
		const float mi = b1 * m[i] + (1.0f - b1) * gi;
		const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
		m[i] = mi;
		v[i] = vi;
		p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	}
}

// Search centres from the predictions: round(pred * 16), clamped to +-range.
__global__ void centers_kernel(const float* __restrict__ pred, int32_t* __restrict__ centers, int n, int range,
                               const umi::MeZero zero) {
	zero.run();
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * n; i += gridDim.x * blockDim.x) {
		const float v = rintf(pred[i] * 16.0f);
		centers[i] = (int32_t)fminf(fmaxf(v, (float)-range), (float)range);
	}
}

// List for the exhaustive search: every block other than the audited ones
// (0, stride, 2 stride, ...) whose refined SAD exceeds the threshold
// (counted in count[1]), and, when `with_audit`, the audited blocks too
// (their refined SAD goes to audit_sums[0]).  count[0] is the list length.
// List order is the order of discovery; the search is per block, so the
// order changes no result.
__global__ void flag_kernel(const int32_t* __restrict__ mv, int n, int stride, int32_t thr, bool with_audit,
                            int32_t* __restrict__ list, int32_t* __restrict__ count,
                            unsigned long long* __restrict__ audit_sums) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		if (stride > 0 && i % stride == 0) {
			if (with_audit) {
				if (audit_sums) atomicAdd(audit_sums, (unsigned long long)mv[3 * i + 2]);
				list[atomicAdd(count, 1)] = i;
			}
		} else if (mv[3 * i + 2] > thr) {
			list[atomicAdd(count, 1)] = i;
			atomicAdd(count + 1, 1);
		}
	}
}

// audit_sums[1] += exhaustive SAD of the audited blocks, searched in the
// same list as the fallback blocks.
__global__ void audit_sum_kernel(const int32_t* __restrict__ mv, int n, int stride,
                                 unsigned long long* __restrict__ audit_sums, const int32_t* __restrict__ fallback,
                                 int32_t* __restrict__ n_fallback) {
	if (n_fallback && blockIdx.x == 0 && threadIdx.x == 0) *n_fallback = *fallback;
	const int na = (n + stride - 1) / stride;
	unsigned long long s = 0;
	for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x)
		s += (unsigned long long)mv[3 * (size_t)a * stride + 2];
	for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	if ((threadIdx.x & 31) == 0 && s) atomicAdd(audit_sums + 1, s);
}

// alist = 0, stride, 2 stride, ... (*acount = their number).
__global__ void audit_list_kernel(int32_t* __restrict__ alist, int32_t* __restrict__ acount, int n, int stride) {
	const int na = (n + stride - 1) / stride;
	for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) alist[a] = a * stride;
	if (blockIdx.x == 0 && threadIdx.x == 0) *acount = na;
}

// The audited blocks take their exhaustive result (amv) in place of the
// refined one (mv); audit_sums (if non-null) += (refined SAD, exhaustive SAD).
__global__ void audit_merge_kernel(int32_t* __restrict__ mv, const int32_t* __restrict__ amv, int n, int stride,
                                   unsigned long long* __restrict__ audit_sums, const int32_t* __restrict__ fallback,
                                   int32_t* __restrict__ n_fallback) {
	if (n_fallback && blockIdx.x == 0 && threadIdx.x == 0) *n_fallback = *fallback;
	const int na = (n + stride - 1) / stride;
	unsigned long long s0 = 0, s1 = 0;
	for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
		const size_t j = 3 * (size_t)a * stride;
		s0 += (unsigned long long)mv[j + 2];
		s1 += (unsigned long long)amv[j + 2];
		mv[j] = amv[j];
		mv[j + 1] = amv[j + 1];
		mv[j + 2] = amv[j + 2];
	}
	if (!audit_sums) return;
	for (int o = 16; o > 0; o >>= 1) {
		s0 += __shfl_xor_sync(0xffffffffu, s0, o);
		s1 += __shfl_xor_sync(0xffffffffu, s1, o);
	}
	if ((threadIdx.x & 31) == 0) {
		if (s0) atomicAdd(audit_sums, s0);
		if (s1) atomicAdd(audit_sums + 1, s1);
	}
}

// ---- tensor-core inference path: bf16 NHWC activations, 32 channels (64
// bytes) per pixel, layers 2-4 on tcgen05 (umi::menet_conv_tc).

// Weights of layers 1..3 as (32, 9*32) bf16 K-major matrices (column
// tap*32 + ci), all three in one launch: blockIdx.y = layer - 1.
static_assert(NL == 4, "pack_tc_weights_kernel selects among three layers");
struct TcWeights {
	const float* w[NL - 1];
	__nv_bfloat16* out[NL - 1];
};
__global__ void pack_tc_weights_kernel(TcWeights p) {
	const int l = blockIdx.y;
	const float* w = l == 0 ? p.w[0] : l == 1 ? p.w[1] : p.w[2];
	__nv_bfloat16* out = l == 0 ? p.out[0] : l == 1 ? p.out[1] : p.out[2];
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < CH * 9 * CH; i += gridDim.x * blockDim.x) {
		const int co = i / (9 * CH), r = i - co * 9 * CH, tap = r / CH, ci = r - tap * CH;
		out[i] = __float2bfloat16_rn(w[(co * CH + ci) * 9 + tap]);
	}
}

// Layer 1 (2 -> 32 channels, dilation 1) on the FP32 pipe: + bias, ReLU,
// bf16, 64-byte NHWC pixels.  Weights come straight from the parameters
// ([co][ci][tap], rounded to bf16 here).  A thread computes one 16-byte
// quarter of the output pixel (8 channels, q = thread & 3) for four adjacent
// pixels x .. x+3 (x a multiple of 4, W a multiple of 4), from a 3 x 6 window
// per input channel: one 16-byte load and two edge loads per window row.
// Each accumulator sums bias, then the 18 products in (ci, tap) order.
__global__ void __launch_bounds__(NT) conv1_nhwc_kernel(const float* __restrict__ x0, const float* __restrict__ w,
                                                        const float* __restrict__ bias, __nv_bfloat16* __restrict__ out,
                                                        int H, int W) {
	__shared__ float4 ws[18][CH / 4];  // [ci * 9 + tap][co / 4]
	__shared__ float4 bs[CH / 4];
	for (int i = threadIdx.x; i < CH * 18; i += NT) {
		const int co = i / 18, k = i - co * 18;
		reinterpret_cast<float*>(ws)[k * CH + co] = __bfloat162float(__float2bfloat16_rn(w[i]));
	}
	if (threadIdx.x < CH) reinterpret_cast<float*>(bs)[threadIdx.x] = bias[threadIdx.x];
	__syncthreads();
	const int P = H * W, groups_x = W >> 2;
	const int t = blockIdx.x * NT + threadIdx.x, q = t & 3, pg = t >> 2;
	if (pg >= H * groups_x) return;
	const int y = pg / groups_x, x = (pg - y * groups_x) * 4;
	float in[2][3][6];
#pragma unroll
	for (int ci = 0; ci < 2; ++ci)
#pragma unroll
		for (int r = 0; r < 3; ++r) {
			const int yy = y + r - 1;
			if (yy >= 0 && yy < H) {
				const float* row = x0 + (size_t)ci * P + (size_t)yy * W + x;
				const float4 m = *reinterpret_cast<const float4*>(row);
				in[ci][r][0] = x > 0 ? row[-1] : 0.0f;
				in[ci][r][1] = m.x; in[ci][r][2] = m.y; in[ci][r][3] = m.z; in[ci][r][4] = m.w;
				in[ci][r][5] = x + 4 < W ? row[4] : 0.0f;
			} else {
#pragma unroll
				for (int c = 0; c < 6; ++c) in[ci][r][c] = 0.0f;
			}
		}
	float acc[4][8];
	{
		const float4 b0 = bs[2 * q], b1 = bs[2 * q + 1];
#pragma unroll
		for (int px = 0; px < 4; ++px) {
			acc[px][0] = b0.x; acc[px][1] = b0.y; acc[px][2] = b0.z; acc[px][3] = b0.w;
			acc[px][4] = b1.x; acc[px][5] = b1.y; acc[px][6] = b1.z; acc[px][7] = b1.w;
		}
	}
#pragma unroll
	for (int ci = 0; ci < 2; ++ci)
#pragma unroll
		for (int tap = 0; tap < 9; ++tap) {
			const float4 wa = ws[ci * 9 + tap][2 * q], wb = ws[ci * 9 + tap][2 * q + 1];
			const float wv[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
			for (int px = 0; px < 4; ++px) {
				const float v = in[ci][tap / 3][px + tap % 3];
#pragma unroll
				for (int c = 0; c < 8; ++c) acc[px][c] = fmaf(wv[c], v, acc[px][c]);
			}
		}
#pragma unroll
	for (int px = 0; px < 4; ++px) {
		uint32_t pk[4];
#pragma unroll
		for (int c2 = 0; c2 < 4; ++c2) {
			const __nv_bfloat162 b2 =
				__floats2bfloat162_rn(fmaxf(acc[px][2 * c2], 0.0f), fmaxf(acc[px][2 * c2 + 1], 0.0f));
			pk[c2] = *reinterpret_cast<const uint32_t*>(&b2);
		}
		*reinterpret_cast<uint4*>(out + ((size_t)y * W + x + px) * CH + q * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
	}
}

// Head on the bf16 NHWC layer-4 activations.  A block's 16 cells are four
// rows of 256 contiguous bytes; a warp reads them as two 16-byte pieces per
// lane (piece j = lane + 32 s: row j >> 4, cell (j >> 2) & 3, channels
// 8 (j & 3) .. +7), so each lane keeps the 32 head weights of its pieces in
// registers for every block it serves.  HEAD_BPW blocks per warp, all their
// loads issued before the first product.
constexpr int HEAD_WARPS = 8, HEAD_BPW = 4;
__global__ void __launch_bounds__(HEAD_WARPS * 32)
	head_nhwc_kernel(const __nv_bfloat16* __restrict__ a4, const float* __restrict__ params, int wh_off, int bh_off,
                     float* __restrict__ pred, int W4, int nbx, int nblk) {
	__shared__ float4 wsm[2][64][2];  // [output][piece][channels 0-3, 4-7 of the piece], bf16-rounded
	for (int t = threadIdx.x; t < 2 * HEADF; t += blockDim.x) {
		const int o = t / HEADF, f = t - o * HEADF, c = f >> 4, cell = f & 15;
		const int j = (cell >> 2) * 16 + (cell & 3) * 4 + (c >> 3);
		reinterpret_cast<float*>(&wsm[o][j][0])[c & 7] = __bfloat162float(__float2bfloat16_rn(params[wh_off + t]));
	}
	__syncthreads();
	const int lane = threadIdx.x & 31;
	const int first = (blockIdx.x * HEAD_WARPS + (threadIdx.x >> 5)) * HEAD_BPW;
	if (first >= nblk) return;
	float wt[2][2][8];  // [output][piece s][channel in the piece]
#pragma unroll
	for (int o = 0; o < 2; ++o)
#pragma unroll
		for (int s = 0; s < 2; ++s) {
			const float4 a = wsm[o][lane + 32 * s][0], b = wsm[o][lane + 32 * s][1];
			wt[o][s][0] = a.x; wt[o][s][1] = a.y; wt[o][s][2] = a.z; wt[o][s][3] = a.w;
			wt[o][s][4] = b.x; wt[o][s][5] = b.y; wt[o][s][6] = b.z; wt[o][s][7] = b.w;
		}
	const size_t row_pieces = (size_t)W4 * CH * sizeof(__nv_bfloat16) / 16;
	uint4 v[HEAD_BPW][2];
#pragma unroll
	for (int u = 0; u < HEAD_BPW; ++u) {
		const int blk = min(first + u, nblk - 1);  // past the end: reload the last block, store nothing
		const int by = blk / nbx, bx = blk - by * nbx;
		const uint4* base = reinterpret_cast<const uint4*>(a4 + ((size_t)(4 * by) * W4 + 4 * bx) * CH) + (lane & 15);
#pragma unroll
		for (int s = 0; s < 2; ++s) v[u][s] = __ldg(base + ((lane >> 4) + 2 * s) * row_pieces);
	}
	const float b0 = params[bh_off], b1 = params[bh_off + 1];
#pragma unroll
	for (int u = 0; u < HEAD_BPW; ++u) {
		float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
		for (int s = 0; s < 2; ++s) {
			const uint32_t word[4] = {v[u][s].x, v[u][s].y, v[u][s].z, v[u][s].w};
#pragma unroll
			for (int e = 0; e < 8; ++e) {
				const float a = __uint_as_float(e & 1 ? word[e >> 1] & 0xffff0000u : word[e >> 1] << 16);
				s0 = fmaf(wt[0][s][e], a, s0);
				s1 = fmaf(wt[1][s][e], a, s1);
			}
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			s0 += __shfl_xor_sync(0xffffffffu, s0, o);
			s1 += __shfl_xor_sync(0xffffffffu, s1, o);
		}
		if (lane == 0 && first + u < nblk)
			*reinterpret_cast<float2*>(pred + 2 * (size_t)(first + u)) = make_float2(s0 + b0, s1 + b1);
	}
}

// ------------------------------------------------------------------ host side
const Layout& layout() {
	static const Layout L;
	return L;
}

umi_status check_frame(int h, int w) {
	if (h < 16 || w < 16) return umi::fail(UMI_ERR_INVALID_ARG, "learned ME: frame %dx%d smaller than one block", h, w);
	if (h % 16 || w % 16) return umi::fail(UMI_ERR_UNSUPPORTED, "learned ME: frame %dx%d not a multiple of 16", h, w);
	return UMI_OK;
}

int grid_for(size_t n) { return (int)std::min<size_t>((n + NT - 1) / NT, 4096); }

template <int DIL>
umi_status conv_dil(const float* in, const float* w, const float* bias, float* out, const Work& K, cudaStream_t st) {
	auto kern = menet_train::conv_kernel<DIL>;
	constexpr int SMEM = (int)menet_train::ConvTile<DIL>::smem;
	UMI_TRY(umi::cuda_status(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
	                         "cudaFuncSetAttribute"));
	kern<<<dim3(umi::ceil_div(K.W4, 32), umi::ceil_div(K.H4, 16)), NT, SMEM, st>>>(in, w, bias, out, K.H4, K.W4);
	return umi::launch_status("conv_kernel");
}

// Layer l = 1, 2, 3 (dilations 2, 4, 8), forward.
umi_status conv_layer(int l, const float* in, const float* w, const float* bias, float* out, const Work& K,
                      cudaStream_t st) {
	static_assert(DIL[1] == 2 && DIL[2] == 4 && DIL[3] == 8, "one instance per layer");
	if (l == 1) return conv_dil<DIL[1]>(in, w, bias, out, K, st);
	if (l == 2) return conv_dil<DIL[2]>(in, w, bias, out, K, st);
	return conv_dil<DIL[3]>(in, w, bias, out, K, st);
}

template <int DIL>
umi_status wgrad_dil(const float* in, const float* dpre, float* part, const Work& K, int units, int per, int grid,
                     cudaStream_t st) {
	auto kern = menet_train::wgrad_kernel<DIL>;
	constexpr int SMEM = (int)menet_train::WgradTile<DIL>::smem;
	UMI_TRY(umi::cuda_status(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
	                         "cudaFuncSetAttribute"));
	kern<<<grid, NT, SMEM, st>>>(in, dpre, part, K.H4, K.W4, units, per);
	return umi::launch_status("wgrad_kernel");
}

// out[0 .. cols) (and *extra, the column after them) = sums of the partial rows.
umi_status reduce_rows(const float* part, float* out, float* extra, int n, int m, int cols, const int32_t* err,
                       int32_t* report, cudaStream_t st) {
	menet_train::reduce_rows_kernel<<<umi::ceil_div(m, 32), NT, 0, st>>>(part, out, extra, n, m, cols, err, report);
	return umi::launch_status("reduce_rows_kernel");
}

umi_status forward(const uint8_t* cur, const uint8_t* ref, int w, const float* params, const Work& K, void* ws,
                   cudaStream_t st) {
	const Layout& L = layout();
	downsample4_kernel<<<grid_for(2 * (size_t)K.P), NT, 0, st>>>(cur, ref, K.at<float>(ws, K.x0), w, K.H4, K.W4);
	UMI_TRY(umi::launch_status("downsample4_kernel"));
	auto pack = [&](int first, int n) {  // the weights of layers first .. first + n - 1
		menet_train::Pack pk{};
		for (int l = first; l < first + n; ++l) {
			pk.w[l] = params + L.w[l];
			pk.fwd[l] = K.at<float>(ws, K.wf[l]);
			pk.bwd[l] = l ? K.at<__nv_bfloat16>(ws, K.wt[l]) : nullptr;
		}
		menet_train::pack_weights_kernel<<<dim3(grid_for(CH * CH * 9), n), NT, 0, st>>>(pk, first);
		return umi::launch_status("pack_weights_kernel");
	};
	UMI_TRY(pack(0, K.whole ? NL : 1));
	menet_train::conv_first_kernel<<<umi::ceil_div(K.P / 4, NT), NT, 0, st>>>(
		K.at<float>(ws, K.x0), K.at<float>(ws, K.wf[0]), params + L.b[0], K.at<float>(ws, K.act[0]), K.H4, K.W4);
	UMI_TRY(umi::launch_status("conv_first_kernel"));
	for (int l = 1; l < NL; ++l) {
		if (!K.whole) UMI_TRY(pack(l, 1));
		UMI_TRY(conv_layer(l, K.at<float>(ws, K.act[l - 1]), K.at<float>(ws, K.wf[l]), params + L.b[l],
		                   K.at<float>(ws, K.act[l]), K, st));
	}
	menet_train::head_fwd_kernel<<<dim3(umi::ceil_div(K.nbx, 64), K.nby), NT, 0, st>>>(
		K.at<float>(ws, K.act[NL - 1]), params + L.wh, params + L.bh, K.at<float>(ws, K.pred), K.H4, K.W4, K.nbx);
	return umi::launch_status("head_fwd_kernel");
}

// Inference forward pass with layers 2-4 on the tensor cores; prediction to K.pred.
umi_status infer(const uint8_t* cur, const uint8_t* ref, int w, const float* params, const Work& K, void* ws, int32_t* err,
                 cudaStream_t st) {
	const Layout& L = layout();
	downsample4_kernel<<<grid_for(2 * (size_t)K.P), NT, 0, st>>>(cur, ref, K.at<float>(ws, K.x0), w, K.H4, K.W4);
	UMI_TRY(umi::launch_status("downsample4_kernel"));
	TcWeights tw;
	for (int l = 1; l < NL; ++l) {
		tw.w[l - 1] = params + L.w[l];
		tw.out[l - 1] = K.at<__nv_bfloat16>(ws, K.wtc[l]);
	}
	pack_tc_weights_kernel<<<dim3(grid_for(CH * 9 * CH), NL - 1), NT, 0, st>>>(tw);
	UMI_TRY(umi::launch_status("pack_tc_weights_kernel"));
	__nv_bfloat16* a = K.at<__nv_bfloat16>(ws, K.nhwc[0]);
	__nv_bfloat16* b = K.at<__nv_bfloat16>(ws, K.nhwc[1]);
	conv1_nhwc_kernel<<<umi::ceil_div(K.P, NT), NT, 0, st>>>(K.at<float>(ws, K.x0), params + L.w[0], params + L.b[0], a,
	                                                         K.H4, K.W4);
	UMI_TRY(umi::launch_status("conv1_nhwc_kernel"));
	for (int l = 1; l < NL; ++l) {
		UMI_TRY(umi::menet_conv_tc(a, b, K.at<__nv_bfloat16>(ws, K.wtc[l]), params + L.b[l], K.H4, K.W4, DIL[l], err, st));
		std::swap(a, b);
	}
	head_nhwc_kernel<<<umi::ceil_div(K.nblk, HEAD_WARPS * HEAD_BPW), HEAD_WARPS * 32, 0, st>>>(
		a, params, L.wh, L.bh, K.at<float>(ws, K.pred), K.W4, K.nbx, K.nblk);
	return umi::launch_status("head_nhwc_kernel");
}

}  // namespace

extern "C" umi_status umi_menet_infer(const uint8_t* cur, const uint8_t* ref, int32_t h, int32_t w, const float* params,
                                      float* pred, int32_t* err, void* workspace, size_t workspace_bytes, void* stream) {
	UMI_TRY(check_frame(h, w));
	if (!cur || !ref || !params || !workspace) return umi::fail(UMI_ERR_INVALID_ARG, "menet_infer: null pointer");
	const Work K(h, w, workspace_bytes);
	if (workspace_bytes < K.least) return umi::fail(UMI_ERR_NO_MEMORY, "menet_infer: workspace too small");
	if (!umi::aligned(workspace, 256)) return umi::fail(UMI_ERR_INVALID_ARG, "menet_infer: workspace alignment");
	const cudaStream_t st = umi::as_stream(stream);
	UMI_TRY(infer(cur, ref, w, params, K, workspace, err, st));
	if (pred)
		UMI_TRY(umi::cuda_status(cudaMemcpyAsync(pred, K.at<float>(workspace, K.pred), sizeof(float) * 2 * K.nblk,
		                                         cudaMemcpyDeviceToDevice, st),
		                         "cudaMemcpyAsync"));
	return umi::ok();
}

extern "C" int32_t umi_menet_param_count(void) { return layout().total; }

extern "C" size_t umi_menet_workspace_bytes(int32_t h, int32_t w) {
	if (check_frame(h, w) != UMI_OK) return 0;
	return Work(h, w).bytes;
}

extern "C" umi_status umi_menet_forward(const uint8_t* cur, const uint8_t* ref, int32_t h, int32_t w, const float* params,
                                        float* pred, void* workspace, size_t workspace_bytes, void* stream) {
	UMI_TRY(check_frame(h, w));
	if (!cur || !ref || !params || !workspace) return umi::fail(UMI_ERR_INVALID_ARG, "menet_forward: null pointer");
	const Work K(h, w, workspace_bytes);
	if (workspace_bytes < K.least) return umi::fail(UMI_ERR_NO_MEMORY, "menet_forward: workspace too small");
	if (!umi::aligned(workspace, 256)) return umi::fail(UMI_ERR_INVALID_ARG, "menet_forward: workspace alignment");
	const cudaStream_t st = umi::as_stream(stream);
	UMI_TRY(forward(cur, ref, w, params, K, workspace, st));
	if (pred)
		UMI_TRY(umi::cuda_status(cudaMemcpyAsync(pred, K.at<float>(workspace, K.pred), sizeof(float) * 2 * K.nblk,
		                                         cudaMemcpyDeviceToDevice, st),
		                         "cudaMemcpyAsync"));
	return umi::ok();
}

extern "C" umi_status umi_menet_backward_err(const int32_t* target, int32_t target_stride, int32_t h, int32_t w,
                                             const float* params, float* grads, float* loss, int32_t* err,
                                             unsigned long long wait_ns, void* workspace, size_t workspace_bytes,
                                             void* stream) {
	UMI_TRY(check_frame(h, w));
	if (!target || !params || !grads || !workspace) return umi::fail(UMI_ERR_INVALID_ARG, "menet_backward: null pointer");
	const Work K(h, w, workspace_bytes);
	if (workspace_bytes < K.least) return umi::fail(UMI_ERR_NO_MEMORY, "menet_backward: workspace too small");
	if (!umi::aligned(workspace, 256)) return umi::fail(UMI_ERR_INVALID_ARG, "menet_backward: workspace alignment");
	const Layout& L = layout();
	const cudaStream_t st = umi::as_stream(stream);
	void* ws = workspace;
	// the gradient in fp32, the same as parts, and a free slot for the next one's
	// fp32 form; its parts replace the fp32 form that the weight gradient has read
	size_t dcur = K.slot[0], din = K.slot[1], dnext = K.slot[2];
	int32_t* bits = K.at<int32_t>(ws, K.err);  // of this pass's waits, cleared by its first kernel
	menet_train::head_bwd_kernel<<<K.head_parts, NT, 0, st>>>(K.at<float>(ws, K.act[NL - 1]), params + L.wh,
	                                                K.at<float>(ws, K.pred), target, target_stride,
	                                                K.at<float>(ws, dcur), K.at<float>(ws, K.part), K.H4, K.W4, K.nbx,
	                                                K.nblk, K.htx, K.htiles, bits);
	UMI_TRY(umi::launch_status("head_bwd_kernel"));
	float* part = K.at<float>(ws, K.part);
	UMI_TRY(reduce_rows(part, grads + L.wh, loss, K.head_parts, 2 * HEADF + 3, 2 * HEADF + 2, bits, nullptr, st));
	UMI_TRY(umi::menet_to_parts(K.at<float>(ws, dcur), K.at<void>(ws, din), K.P, st));
	const int units = K.units, per = umi::ceil_div(units, K.parts), grid = umi::ceil_div(units, per);
	for (int l = NL - 1; l >= 0; --l) {
		const float* in = l == 0 ? K.at<float>(ws, K.x0) : K.at<float>(ws, K.act[l - 1]);
		const float* d = K.at<float>(ws, dcur);
		const int m = CH * CIN[l] * 9 + CH;
		if (l == 3) UMI_TRY(wgrad_dil<DIL[3]>(in, d, part, K, units, per, grid, st));
		else if (l == 2) UMI_TRY(wgrad_dil<DIL[2]>(in, d, part, K, units, per, grid, st));
		else if (l == 1) UMI_TRY(wgrad_dil<DIL[1]>(in, d, part, K, units, per, grid, st));
		else {
			menet_train::wgrad_first_kernel<<<grid, NT, 0, st>>>(in, d, part, K.H4, K.W4, units, per);
			UMI_TRY(umi::launch_status("wgrad_first_kernel"));
		}
		// grads[w_l], then grads[b_l] right after it (same layout as the partial rows)
		UMI_TRY(reduce_rows(part, grads + L.w[l], nullptr, grid, m, m, bits, l == 0 ? err : nullptr, st));
		if (l > 0) {  // data gradient, masked by ReLU(a_{l-1})
			UMI_TRY(umi::menet_dgrad(K.at<void>(ws, din), K.at<void>(ws, K.wt[l]), K.at<float>(ws, K.act[l - 1]),
			                         K.at<float>(ws, dnext), l > 1 ? K.at<void>(ws, dcur) : nullptr, K.H4, K.W4, DIL[l],
			                         bits, wait_ns, st));
			const size_t read = din;
			din = dcur;
			dcur = dnext;
			dnext = read;
		}
	}
	return umi::ok();
}

extern "C" umi_status umi_menet_backward(const int32_t* target, int32_t target_stride, int32_t h, int32_t w,
                                         const float* params, float* grads, float* loss, void* workspace,
                                         size_t workspace_bytes, void* stream) {
	return umi_menet_backward_err(target, target_stride, h, w, params, grads, loss, nullptr, 0, workspace, workspace_bytes,
	                              stream);
}

extern "C" umi_status umi_menet_adam(float* params, const float* grads, float* m, float* v, int32_t step, float lr,
                                     void* stream) {
	if (!params || !grads || !m || !v || step < 1) return umi::fail(UMI_ERR_INVALID_ARG, "menet_adam: bad arguments");
	const int n = layout().total;
	const float b1 = 0.9f, b2 = 0.999f;
	const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
	adam_kernel<<<grid_for(n), NT, 0, umi::as_stream(stream)>>>(params, grads, m, v, n, lr, b1, b2, 1e-8f, c1, c2);
	UMI_TRY(umi::launch_status("adam_kernel"));
	return umi::ok();
}

extern "C" umi_status umi_me_learned_u8(const uint8_t* cur, const uint8_t* ref, int32_t h, int32_t w, const float* params,
                                        int32_t refine_r, int32_t full_r, int32_t sad_threshold, int32_t audit_stride,
                                        int32_t* mv, unsigned long long* audit_sums, int32_t* n_fallback,
                                        void* workspace, size_t workspace_bytes, void* stream) {
	UMI_TRY(check_frame(h, w));
	if (!cur || !ref || !params || !mv || !workspace) return umi::fail(UMI_ERR_INVALID_ARG, "me_learned: null pointer");
	const Work K(h, w, workspace_bytes);
	if (workspace_bytes < K.least) return umi::fail(UMI_ERR_NO_MEMORY, "me_learned: workspace too small");
	if (!umi::aligned(workspace, 256)) return umi::fail(UMI_ERR_INVALID_ARG, "me_learned: workspace alignment");
	if (refine_r < 1 || full_r < refine_r || full_r > 64)
		return umi::fail(UMI_ERR_UNSUPPORTED, "me_learned: refine %d / full %d ranges", refine_r, full_r);
	if (audit_stride < 0) return umi::fail(UMI_ERR_INVALID_ARG, "me_learned: negative audit stride");
	const cudaStream_t st = umi::as_stream(stream);
	void* ws = workspace;
	const umi::MeFinishBuffers fb{K.at<int32_t>(ws, K.list), K.at<int32_t>(ws, K.count), K.at<int32_t>(ws, K.alist),
	                              K.at<int32_t>(ws, K.amv)};
	umi::MeAudit audit;
	UMI_TRY(umi::me_audit_begin(cur, ref, h, w, full_r, audit_stride, fb, st, &audit));
	UMI_TRY(infer(cur, ref, w, params, K, ws, K.at<int32_t>(ws, K.err), st));
	int32_t* centers = K.at<int32_t>(ws, K.centers);
	centers_kernel<<<grid_for(2 * (size_t)K.nblk), NT, 0, st>>>(K.at<float>(ws, K.pred), centers, K.nblk,
	                                                             full_r - refine_r, umi::MeZero{fb.count, audit_sums});
	UMI_TRY(umi::launch_status("centers_kernel"));
	return umi::me_refine_fallback_finish(cur, ref, h, w, centers, refine_r, full_r, sad_threshold, audit_stride, mv,
	                                      audit_sums, n_fallback, fb, audit, st);
}

namespace umi {

namespace {

// The calling thread's second stream on one device, with its fork and join
// events: made on first use outside a stream capture, destroyed at thread exit.
struct AuxStream {
	cudaStream_t s = nullptr;
	cudaEvent_t fork = nullptr, join = nullptr;
	~AuxStream() {
		if (join) cudaEventDestroy(join);
		if (fork) cudaEventDestroy(fork);
		if (s) cudaStreamDestroy(s);
	}
};

AuxStream* aux_stream(cudaStream_t st) {
	constexpr int kMaxDevices = 64;
	thread_local AuxStream aux[kMaxDevices];
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
	AuxStream& a = aux[dev];
	if (a.s && a.fork && a.join) return &a;
	cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
	if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
		cudaGetLastError();  // not an error of this call: the stage runs in order on st
		return nullptr;
	}
	if (cs != cudaStreamCaptureStatusNone) return nullptr;
	if (!a.s && cudaStreamCreateWithFlags(&a.s, cudaStreamNonBlocking) != cudaSuccess) a.s = nullptr;
	if (!a.fork && cudaEventCreateWithFlags(&a.fork, cudaEventDisableTiming) != cudaSuccess) a.fork = nullptr;
	if (!a.join && cudaEventCreateWithFlags(&a.join, cudaEventDisableTiming) != cudaSuccess) a.join = nullptr;
	cudaGetLastError();  // a failure here only means no second stream
	return a.s && a.fork && a.join ? &a : nullptr;
}

}  // namespace

umi_status me_audit_begin(const uint8_t* cur, const uint8_t* ref, int h, int w, int full_r, int audit_stride,
                          const MeFinishBuffers& b, cudaStream_t st, MeAudit* audit) {
	audit->active = audit->combined = audit->forked = audit->joined = false;
	audit->done = nullptr;
	audit->st = st;
	const int nblk = (h / 16) * (w / 16);
	if (audit_stride <= 0 || nblk == 0) return UMI_OK;
	audit->active = true;
	// A +-64 list search runs one block per SM at a time.  An audit of fewer
	// blocks than SMs leaves room in the fallback search's round, so it joins
	// that list; a larger one runs apart, beside the proposal.
	const int na = ceil_div(nblk, audit_stride);
	int dev = 0, sms = 0;
	UMI_TRY(cuda_status(cudaGetDevice(&dev), "cudaGetDevice"));
	UMI_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute"));
	if (na < sms) {
		audit->combined = true;
		return UMI_OK;
	}
	AuxStream* aux = aux_stream(st);
	cudaStream_t as = st;
	if (aux) {
		UMI_TRY(cuda_status(cudaEventRecord(aux->fork, st), "cudaEventRecord"));
		UMI_TRY(cuda_status(cudaStreamWaitEvent(aux->s, aux->fork, 0), "cudaStreamWaitEvent"));
		as = aux->s;
	}
	audit_list_kernel<<<grid_for(na), NT, 0, as>>>(b.alist, b.count + 2, nblk, audit_stride);
	umi_status rc = launch_status("audit_list_kernel");
	if (rc == UMI_OK)
		rc = umi_full_me_u8_list(cur, ref, h, w, 16, full_r, nullptr, b.alist, b.count + 2, na, b.amv, as);
	if (aux) {
		// recorded on every path once the fork happened: whatever was issued on
		// the second stream is joined back into the caller's stream
		const umi_status jr = cuda_status(cudaEventRecord(aux->join, aux->s), "cudaEventRecord");
		if (jr == UMI_OK) {
			audit->forked = true;
			audit->done = aux->join;
		} else {
			cudaStreamSynchronize(aux->s);  // no join event: the second stream's work ends here
			if (rc == UMI_OK) rc = jr;
		}
	}
	return rc;
}

// Refine around the proposal's centres, exhaustive search for every
// non-audited block whose refined SAD exceeds sad_threshold, then the
// audited blocks' exhaustive results (begun by me_audit_begin) replace the
// refined ones.  Shared by the learned and the coarse proposal.
umi_status me_refine_fallback_finish(const uint8_t* cur, const uint8_t* ref, int h, int w, const int32_t* centers,
                                     int refine_r, int full_r, int32_t sad_threshold, int audit_stride, int32_t* mv,
                                     unsigned long long* audit_sums, int32_t* n_fallback, const MeFinishBuffers& b,
                                     const MeAudit& audit, cudaStream_t st) {
	const int nblk = (h / 16) * (w / 16);
	void* stream = st;
	UMI_TRY(umi_full_me_u8(cur, ref, h, w, 16, refine_r, centers, mv, stream));
	flag_kernel<<<grid_for(nblk), NT, 0, st>>>(mv, nblk, audit.active ? audit_stride : 0, sad_threshold, audit.combined,
	                                           b.list, b.count, audit_sums);
	UMI_TRY(launch_status("flag_kernel"));
	UMI_TRY(umi_full_me_u8_list(cur, ref, h, w, 16, full_r, nullptr, b.list, b.count, nblk, mv, stream));
	if (audit.combined && audit_sums) {
		audit_sum_kernel<<<grid_for(ceil_div(nblk, audit_stride)), NT, 0, st>>>(mv, nblk, audit_stride, audit_sums,
		                                                                        b.count + 1, n_fallback);
		UMI_TRY(launch_status("audit_sum_kernel"));
		n_fallback = nullptr;  // written
	} else if (audit.active && !audit.combined) {
		if (audit.forked) {
			UMI_TRY(cuda_status(cudaStreamWaitEvent(st, audit.done, 0), "cudaStreamWaitEvent"));
			audit.joined = true;
		}
		audit_merge_kernel<<<grid_for(ceil_div(nblk, audit_stride)), NT, 0, st>>>(mv, b.amv, nblk, audit_stride,
		                                                                          audit_sums, b.count + 1, n_fallback);
		UMI_TRY(launch_status("audit_merge_kernel"));
		n_fallback = nullptr;  // written
	}
	if (n_fallback)
		UMI_TRY(cuda_status(cudaMemcpyAsync(n_fallback, b.count + 1, sizeof(int32_t), cudaMemcpyDeviceToDevice, st),
		                    "cudaMemcpyAsync"));
	return ok();
}

}  // namespace umi
