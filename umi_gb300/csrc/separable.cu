// Separable window sum of a float image (a Gaussian blur, for instance), both
// passes in one launch, sm_103a:
//   tmp[y][x] = sum_i w[i] in[y][x + i - k/2],  out[y][x] = sum_i w[i] tmp[y + i - k/2][x],
// i ascending, one fma each, coordinates clamped to the image: the bits of the
// two window sums through umi_launch.
//
// A CTA stages the halo tile of 128 x 32 outputs, filters its 32 + k - 1 rows
// across into a second tile, then down, 4 x 4 outputs a thread.  The first pass
// is done (32 + k - 1) / 32 times over (1.4 at k = 13), which costs less than
// writing and reading the image between two launches.
// 1080p, 13 weights, cold caches: 12.1 us where the two launches took 9.5 and
// 8.9; from the host 24 -> 18 us a blur.  Bound by issue slots (55 %) and the
// shared-memory loads of the second pass; the bytes take 2.5 us (3.7 with tmp).
#include "common.h"
#include "window_ops.cuh"

namespace {

using umi_window::Image;
using umi_window::NT;
using umi_window::RY;
using umi_window::TX;
using umi_window::TY;

struct SepArgs {
	Image<float> img;
	const float* wts;
	float *tmp, *out;  // tmp may be null
	int h, w, k, tw;
	int vec;           // rows of out (and tmp) are 16-byte aligned
};

__device__ __forceinline__ void store4(float* row, int x, int w, int vec, const float (&v)[4]) {
	if (vec && x + 3 < w) {
		*reinterpret_cast<float4*>(row + x) = make_float4(v[0], v[1], v[2], v[3]);
	} else {
#pragma unroll
		for (int i = 0; i < 4; ++i)
			if (x + i < w) row[x + i] = v[i];
	}
}

// K: taps when known at compile time, else 0.
template <int K>
__global__ void __launch_bounds__(NT) separable_kernel(const SepArgs a) {
	extern __shared__ __align__(16) float sm[];
	const int k = K ? K : a.k, rows = TY + k - 1;
	float* tile = sm;                  // [rows][tw]
	float* mid = tile + rows * a.tw;   // [rows][TX]
	float* ws = mid + rows * TX;       // [k]
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
	umi_window::stage_tile(a.img, tile, a.tw, rows, x0 + a.img.ox, y0 + a.img.oy, min(TY, a.h - y0) + k - 1,
	                       min(TX, a.w - x0) + k - 1, warp, lane);
	for (int i = threadIdx.x; i < k; i += NT) ws[i] = __ldg(a.wts + i);
	asm volatile("cp.async.wait_all;" ::: "memory");
	__syncthreads();
	const int x = x0 + 4 * lane;
	for (int r = warp; r < rows; r += NT / 32) {
		const float* p = tile + r * a.tw + 4 * lane;
		float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
		float4 lo = *reinterpret_cast<const float4*>(p);
#pragma unroll
		for (int b = 0; b < k; b += 4) {
			const float4 hi = *reinterpret_cast<const float4*>(p + b + 4);
			const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
			lo = hi;
#pragma unroll
			for (int q = 0; q < 4; ++q)
				if (b + q < k) {
					const float wt = ws[b + q];
#pragma unroll
					for (int i = 0; i < 4; ++i) acc[i] = fmaf(v[q + i], wt, acc[i]);
				}
		}
		*reinterpret_cast<float4*>(mid + r * TX + 4 * lane) = make_float4(acc[0], acc[1], acc[2], acc[3]);
		const int y = y0 + r - k / 2;  // the tile's own rows
		if (a.tmp && y >= y0 && y < min(y0 + TY, a.h)) store4(a.tmp + (size_t)y * a.w, x, a.w, a.vec, acc);
	}
	__syncthreads();
	const int yb = y0 + warp * RY;
	if (x >= a.w || yb >= a.h) return;
	float acc[RY][4] = {};
	const float* p = mid + warp * RY * TX + 4 * lane;
#pragma unroll
	for (int i = 0; i < k + RY - 1; ++i, p += TX) {
		const float4 t = *reinterpret_cast<const float4*>(p);
		const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
		for (int j = 0; j < RY; ++j)
			if (i - j >= 0 && i - j < k) {
				const float wt = ws[i - j];
#pragma unroll
				for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(v[c], wt, acc[j][c]);
			}
	}
#pragma unroll
	for (int j = 0; j < RY; ++j)
		if (yb + j < a.h) store4(a.out + (size_t)(yb + j) * a.w, x, a.w, a.vec, acc[j]);
}

template <int K>
umi_status launch(const SepArgs& a, dim3 grid, size_t smem, cudaStream_t st) {
	UMI_TRY(umi::allow_shared(separable_kernel<K>, smem));
	separable_kernel<K><<<grid, NT, smem, st>>>(a);
	return umi::launch_status("separable_kernel");
}

// Centred windows have an odd number of taps: an instance each up to the
// largest (2160 x 3840, us from the host, with loops of run-time length and so:
// 9 taps 29.5 and 23.0, 19 taps 45 and 35, 31 taps 68 and 51).  Other numbers
// take the loops.
template <int K>
umi_status launch_taps(const SepArgs& a, dim3 grid, size_t smem, cudaStream_t st) {
	if (a.k == K) return launch<K>(a, grid, smem, st);
	if constexpr (K + 2 <= UMI_SEPARABLE_MAX_TAPS) return launch_taps<K + 2>(a, grid, smem, st);
	return launch<0>(a, grid, smem, st);
}

}  // namespace

extern "C" umi_status umi_separable_f32(const float* in, const float* weights, int32_t k, int32_t h, int32_t w, float* tmp,
                                        float* out, void* stream) {
	if (h < 0 || w < 0 || k < 1) return umi::fail(UMI_ERR_INVALID_ARG, "separable: %dx%d image, %d weights", h, w, k);
	if (h == 0 || w == 0) return umi::ok();
	if (!in || !weights || !out) return umi::fail(UMI_ERR_INVALID_ARG, "separable: null pointer");
	SepArgs a{};
	a.img.p = in;
	a.img.h = h; a.img.w = w;
	a.img.oy = a.img.ox = -(k / 2);
	a.wts = weights;
	a.tmp = tmp; a.out = out;
	a.h = h; a.w = w; a.k = k;
	if (k > UMI_SEPARABLE_MAX_TAPS || umi::ceil_div(h, TY) > 65535)
		return umi::fail(UMI_ERR_UNSUPPORTED, "separable: %d weights, %d rows (at most %d, %d)", k, h, UMI_SEPARABLE_MAX_TAPS,
		                 65535 * TY);
	a.tw = TX + ((k + 3) & ~3);
	a.vec = w % 4 == 0 && umi::aligned(out, 16) && umi::aligned(tmp, 16);
	const size_t rows = TY + k - 1, smem = sizeof(float) * (rows * a.tw + rows * TX + k);
	const dim3 grid(umi::ceil_div(w, TX), umi::ceil_div(h, TY));
	const cudaStream_t st = umi::as_stream(stream);
	const umi_status s = launch_taps<3>(a, grid, smem, st);
	return s == UMI_OK ? umi::ok() : s;
}
