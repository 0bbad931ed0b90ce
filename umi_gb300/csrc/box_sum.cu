// Sums of a uint8 image over (2r+1)^2 windows clipped to the image: the integral
// image, then the four corners of every window straight from it, sm_103a.
//   out[y][x] = S(y1, x1) - S(y1, x0) - S(y0, x1) + S(y0, x0),
// y0 = max(y - r, 0), y1 = min(y + r + 1, h), S(y, x) = the sum of the first y
// rows' first x pixels = ii[y - 1][x - 1], 0 at y = 0 or x = 0.
//
// The corner kernel is bound by latency and the 12 bytes a pixel it moves (four
// coalesced reads, three of them from L1 or L2, one write; 16 with J).  Before,
// the integral image was copied into a zero-bordered J and the corners read by a
// window sum over it: 1080p 19.0 us in graph replays and 37 from the host, now
// 13.8 and 20.
#include "common.h"

namespace {

constexpr int NT = 256, PX = 4;  // threads; pixels per thread, 32 columns apart

__global__ void __launch_bounds__(NT) box_corners_kernel(const int32_t* __restrict__ ii, int32_t* __restrict__ J,
                                                         int32_t* __restrict__ out, int h, int w, int r) {
	const int y = blockIdx.y * (NT / 32) + (threadIdx.x >> 5), x = blockIdx.x * 32 * PX + (threadIdx.x & 31);
	if (y >= h) return;
	const int y0 = max(y - r, 0), y1 = min(y + r + 1, h);
	const int32_t* lo = ii + (size_t)(y0 - 1) * w - 1;  // read where y0 > 0 and the column is > 0
	const int32_t* hi = ii + (size_t)(y1 - 1) * w - 1;
	uint32_t s[PX];
#pragma unroll
	for (int k = 0; k < PX; ++k) {
		const int xk = x + 32 * k, x0 = max(xk - r, 0), x1 = min(xk + r + 1, w);
		s[k] = 0;
		if (xk < w) {
			s[k] = (uint32_t)__ldg(hi + x1);
			if (x0 > 0) s[k] -= (uint32_t)__ldg(hi + x0);
			if (y0 > 0) s[k] -= (uint32_t)__ldg(lo + x1);
			if (x0 > 0 && y0 > 0) s[k] += (uint32_t)__ldg(lo + x0);
		}
	}
#pragma unroll
	for (int k = 0; k < PX; ++k) {
		const int xk = x + 32 * k;
		if (xk >= w) break;
		out[(size_t)y * w + xk] = (int32_t)s[k];
		if (J) J[(size_t)(y + 1) * (w + 1) + xk + 1] = __ldg(ii + (size_t)y * w + xk);
	}
}

}  // namespace

extern "C" umi_status umi_box_sum_u8(const uint8_t* in, int32_t h, int32_t w, int32_t radius, int32_t* ii, int32_t* J,
                                     int32_t* out, void* workspace, size_t workspace_bytes, void* stream) {
	if (radius < 0 || radius > (1 << 20)) return umi::fail(UMI_ERR_INVALID_ARG, "box_sum: radius %d", radius);
	if (h > 0 && w > 0 && !out) return umi::fail(UMI_ERR_INVALID_ARG, "box_sum: null pointer");
	const int rows = umi::ceil_div(h, NT / 32);
	if (rows > 65535) return umi::fail(UMI_ERR_UNSUPPORTED, "box_sum: %d rows (at most %d)", h, 65535 * (NT / 32));
	UMI_TRY(umi_iimg_u8_i32(in, ii, h, w, workspace, workspace_bytes, stream));
	if (h == 0 || w == 0) return umi::ok();
	box_corners_kernel<<<dim3(umi::ceil_div(w, 32 * PX), rows), NT, 0, umi::as_stream(stream)>>>(ii, J, out, h, w, radius);
	const umi_status s = umi::launch_status("box_corners_kernel");
	return s == UMI_OK ? umi::ok() : s;
}
