// 2-D window operators behind umi_launch: the plans whose P space is an image
// (h, w), whose A space is a (ky, kx) window walked row-major in one block,
// and whose Loop input is an image read at (y + a_y sy + oy, x + a_x sx + ox)
// (optionally with a weight per window element), one output per pixel.
// generic_launch.cu tries them before the generic kernel: same reads (clamp
// and PAD per dimension), same accumulation order, so the same bits.
//
// The generic kernel spends its time on address arithmetic and loop control
// (53 us for a 5x5 census of a 1080p frame whose bytes take 2.4 us).  Here:
//
//  window_kernel (sx = sy = 1): a CTA stages the halo tile of 128 x 32 outputs
//  in shared memory once (4-byte cp.async, coalesced rows, clamped), then a
//  thread computes 4 x 4 outputs: each window row is read by 16-byte loads
//  that four outputs across and four output rows share.  Bound: issue slots
//  of the strategy itself.
//
//  strided_kernel (any stride): 4 pixels per thread, 32 columns apart, read
//  straight from global memory; clamps only where the window of the CTA's
//  rows and columns can leave the image.
//
// Measured at 1080p: see window_launch().
#pragma once
#include <algorithm>
#include <cstring>

#include "common.h"
#include "umi/UMI_gpu.h"

namespace umi_window {

// ---- the strategies as per-element operations.  T: element type; acc(x, w)
// in window order; begin(centre, constant) and end(constant).
struct Census {
	using T = int;
	static constexpr bool kWeights = false, kCentre = true;
	struct C { int unused; };
	struct Acc { uint32_t bits; int centre; };
	__device__ static Acc begin(int centre, const C&) { return {0u, centre}; }
	// bits = 2 bits + (x < centre): with both sides moved by 2^31 to unsigned,
	// x < c is the carry of c + ~x, added by the second instruction
	__device__ static void step(Acc& a, int x, int) {
		asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %2;\n\taddc.u32 %0, %0, %0;\n\t}"
		    : "+r"(a.bits)
		    : "r"((uint32_t)a.centre ^ 0x80000000u), "r"((uint32_t)x ^ 0x7fffffffu));
	}
	__device__ static int end(const Acc& a, const C&) { return (int)a.bits; }
};
template <bool MAX> struct Extremum {
	using T = int;
	static constexpr bool kWeights = false, kCentre = false;
	struct C { int init; };
	struct Acc { int t; };
	__device__ static Acc begin(int, const C& c) { return {c.init}; }
	__device__ static void step(Acc& a, int x, int) { a.t = MAX ? max(a.t, x) : min(a.t, x); }
	__device__ static int end(const Acc& a, const C&) { return a.t; }
};
struct NeighbourSum {
	using T = int;
	static constexpr bool kWeights = false, kCentre = false;
	struct C { int init, mul; };
	struct Acc { int t; };
	__device__ static Acc begin(int, const C& c) { return {c.init}; }
	__device__ static void step(Acc& a, int x, int) { a.t += x; }
	__device__ static int end(const Acc& a, const C& c) { return a.t * c.mul; }
};
struct WeightedI {
	using T = int;
	static constexpr bool kWeights = true, kCentre = false;
	struct C { int init; };
	struct Acc { int t; };
	__device__ static Acc begin(int, const C& c) { return {c.init}; }
	__device__ static void step(Acc& a, int x, int w) { a.t += x * w; }
	__device__ static int end(const Acc& a, const C&) { return a.t; }
};
struct WeightedF {
	using T = float;
	static constexpr bool kWeights = true, kCentre = false;
	struct C { float init; };
	struct Acc { float t; };
	__device__ static Acc begin(float, const C& c) { return {c.init}; }
	__device__ static void step(Acc& a, float x, float w) { a.t = fmaf(x, w, a.t); }
	__device__ static float end(const Acc& a, const C&) { return a.t; }
};

// An image input: element (y, x) of the point is in[clamp(y + oy)][clamp(x + ox)],
// or pad where a clamped dimension is PAD.
template <class T> struct Image {
	const T* p;
	int h, w, oy, ox;
	int pad_y, pad_x;  // dimension is PAD
	T pad;
	__device__ __forceinline__ T at(int y, int x) const {
		const int cy = min(max(y, 0), h - 1), cx = min(max(x, 0), w - 1);
		if ((pad_y && cy != y) || (pad_x && cx != x)) return pad;
		return __ldg(p + (size_t)cy * w + cx);
	}
};

template <class Op> struct Args {
	using T = typename Op::T;
	Image<T> img, centre;
	const T* wts;   // weight of element (a_y, a_x): wts[a_y wsy + a_x wsx]
	int wsy, wsx;
	T* out;         // pixel (y, x): out[y orow + x]
	int64_t orow;
	int vec;        // rows of out are 16-byte aligned
	int h, w, ky, kx, sy, sx;
	int tw;         // columns of the staged tile
	int cy, cx;     // the centre's place in the tile, from the window's first element; cy < 0: not in it
	typename Op::C c;
};

constexpr int NT = 256, TX = 128, RY = 4, TY = (NT / 32) * RY;

__device__ __forceinline__ void copy4(void* dst, const void* src) {
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// rows x tw elements of im from (ys, xs) by cp.async (the caller waits).  Where
// the tile leaves the image only the urows x ucols that its outputs use: a tile
// of one output column would copy the edge pixel to 131 places of every row,
// one lane after the other (1080 x 1921, dilation 3x3 10.7 -> 6.5 us, 13-tap
// blur 16.0 -> 10.5).
template <class T>
__device__ __forceinline__ void stage_tile(const Image<T>& im, T* tile, int tw, int rows, int xs, int ys, int urows,
                                           int ucols, int warp, int lane) {
	if (xs >= 0 && xs + tw <= im.w && ys >= 0 && ys + rows <= im.h) {
		const T* src = im.p + (size_t)(ys + warp) * im.w + xs + lane;
		T* dst = tile + warp * tw + lane;
		for (int r = warp; r < rows; r += NT / 32) {
#pragma unroll
			for (int c = 0; c < TX; c += 32) copy4(dst + c, src + c);
			for (int c = TX; c < tw - lane; c += 32) copy4(dst + c, src + c);
			src += (size_t)(NT / 32) * im.w;
			dst += (NT / 32) * tw;
		}
	} else {
		for (int r = warp; r < urows; r += NT / 32) {
			const int y = ys + r, cy = min(max(y, 0), im.h - 1);
			const bool yout = im.pad_y && cy != y;
			const T* row = im.p + (size_t)cy * im.w;
			T* dst = tile + (size_t)r * tw;
			for (int c = lane; c < ucols; c += 32) {
				const int x = xs + c, cx = min(max(x, 0), im.w - 1);
				if (yout || (im.pad_x && cx != x)) dst[c] = im.pad;
				else copy4(dst + c, row + cx);
			}
		}
	}
}

// KX: window columns when known at compile time, else 0 (any number, four at a time).
template <class Op, int KX>
__global__ void __launch_bounds__(NT) window_kernel(const Args<Op> a) {
	using T = typename Op::T;
	struct alignas(16) T4 { T v[4]; };
	extern __shared__ __align__(16) unsigned char smem[];
	T* tile = reinterpret_cast<T*>(smem);               // [TY + ky - 1][tw]
	T* ws = tile + (size_t)(TY + a.ky - 1) * a.tw;      // [ky][kxp]: weights, rows padded to four
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, kx = KX ? KX : a.kx, kxp = (kx + 3) & ~3;
	const Image<T>& im = a.img;
	const int rows = TY + a.ky - 1, xs = x0 + im.ox, ys = y0 + im.oy;
	stage_tile(im, tile, a.tw, rows, xs, ys, min(TY, a.h - y0) + a.ky - 1, min(TX, a.w - x0) + kx - 1, warp, lane);
	if (Op::kWeights)
		for (int i = threadIdx.x; i < a.ky * kx; i += NT) {
			const int ay = i / kx, ax = i - ay * kx;
			ws[ay * kxp + ax] = __ldg(a.wts + ay * a.wsy + ax * a.wsx);
		}
	asm volatile("cp.async.wait_all;" ::: "memory");
	__syncthreads();
	const int x = x0 + 4 * lane, yb = y0 + warp * RY;
	if (x >= a.w || yb >= a.h) return;
	typename Op::Acc acc[RY][4];
#pragma unroll
	for (int j = 0; j < RY; ++j)
#pragma unroll
		for (int k = 0; k < 4; ++k)
			acc[j][k] = Op::begin(!Op::kCentre  ? T(0)
			                      : a.cy >= 0 ? tile[(warp * RY + j + a.cy) * a.tw + 4 * lane + k + a.cx]
			                                  : a.centre.at(yb + j + a.centre.oy, x + k + a.centre.ox),
			                      a.c);
	const T* col = tile + (size_t)(warp * RY) * a.tw + 4 * lane;
	if (KX) {
		constexpr int K = KX ? KX : 1, NQ = (K + 6) / 4, NW = (K + 3) / 4;
		// staged row i meets window row i - j of output row j
		auto row = [&](int i, auto checked) {
			T v[4 * NQ];
#pragma unroll
			for (int q = 0; q < NQ; ++q) {
				const T4 t = *reinterpret_cast<const T4*>(col + 4 * q);
#pragma unroll
				for (int k = 0; k < 4; ++k) v[4 * q + k] = t.v[k];
			}
			col += a.tw;
#pragma unroll
			for (int j = 0; j < RY; ++j) {
				const int t = i - j;
				if (decltype(checked)::value && (t < 0 || t >= a.ky)) continue;
				T w[4 * NW] = {};
				if (Op::kWeights)
#pragma unroll
					for (int q = 0; q < NW; ++q) {
						const T4 u = *reinterpret_cast<const T4*>(ws + t * kxp + 4 * q);
#pragma unroll
						for (int k = 0; k < 4; ++k) w[4 * q + k] = u.v[k];
					}
#pragma unroll
				for (int q = 0; q < K; ++q)
#pragma unroll
					for (int k = 0; k < 4; ++k) Op::step(acc[j][k], v[q + k], w[q]);
			}
		};
		int i = 0;
		for (; i < min(RY - 1, a.ky + RY - 1); ++i) row(i, std::true_type());
#pragma unroll 2
		for (; i < a.ky; ++i) row(i, std::false_type());
		for (; i < a.ky + RY - 1; ++i) row(i, std::true_type());
	} else {
		for (int i = 0; i < a.ky + RY - 1; ++i, col += a.tw) {
			T4 lo = *reinterpret_cast<const T4*>(col);
			for (int kb = 0; kb < kx; kb += 4) {
				const T4 hi = *reinterpret_cast<const T4*>(col + kb + 4);
				T v[8];
#pragma unroll
				for (int k = 0; k < 4; ++k) { v[k] = lo.v[k]; v[4 + k] = hi.v[k]; }
				lo = hi;
				const int n = kx - kb;  // window columns left
#pragma unroll
				for (int j = 0; j < RY; ++j) {
					const int t = i - j;
					if (t < 0 || t >= a.ky) continue;
					T4 w = {};
					if (Op::kWeights) w = *reinterpret_cast<const T4*>(ws + t * kxp + kb);
#pragma unroll
					for (int q = 0; q < 4; ++q)
						if (q < n)
#pragma unroll
							for (int k = 0; k < 4; ++k) Op::step(acc[j][k], v[q + k], w.v[q]);
				}
			}
		}
	}
#pragma unroll
	for (int j = 0; j < RY; ++j) {
		if (yb + j >= a.h) break;
		T* o = a.out + (yb + j) * a.orow + x;
		T4 r;
#pragma unroll
		for (int k = 0; k < 4; ++k) r.v[k] = Op::end(acc[j][k], a.c);
		if (a.vec && x + 3 < a.w) {
			*reinterpret_cast<T4*>(o) = r;
		} else {
#pragma unroll
			for (int k = 0; k < 4; ++k)
				if (x + k < a.w) o[k] = r.v[k];
		}
	}
}

// Any stride: thread = pixels x, x + 32, x + 64, x + 96 of one row.
template <class Op>
__global__ void __launch_bounds__(NT) strided_kernel(const Args<Op> a) {
	using T = typename Op::T;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int x = blockIdx.x * TX + lane, y = blockIdx.y * (NT / 32) + warp;
	if (y >= a.h) return;
	const Image<T>& im = a.img;
	const int cx0 = blockIdx.x * TX + im.ox, cy0 = y + im.oy;
	const int ex = (a.kx - 1) * a.sx, ey = (a.ky - 1) * a.sy;
	// every pixel of the warp inside the image at every window element
	const bool inside = cx0 + min(ex, 0) >= 0 && cx0 + TX - 1 + max(ex, 0) < im.w && cy0 + min(ey, 0) >= 0 &&
	                    cy0 + max(ey, 0) < im.h;
	typename Op::Acc acc[4];
#pragma unroll
	for (int k = 0; k < 4; ++k)
		acc[k] = Op::begin(Op::kCentre ? a.centre.at(y + a.centre.oy, x + 32 * k + a.centre.ox) : T(0), a.c);
	for (int ay = 0; ay < a.ky; ++ay)
		for (int ax = 0; ax < a.kx; ++ax) {
			const T w = Op::kWeights ? __ldg(a.wts + ay * a.wsy + ax * a.wsx) : T(0);
			const int yy = cy0 + ay * a.sy, xx = x + im.ox + ax * a.sx;
			T v[4];
			if (inside) {
				const T* p = im.p + (size_t)yy * im.w + xx;
#pragma unroll
				for (int k = 0; k < 4; ++k) v[k] = __ldg(p + 32 * k);
			} else {
#pragma unroll
				for (int k = 0; k < 4; ++k) v[k] = im.at(yy, xx + 32 * k);
			}
#pragma unroll
			for (int k = 0; k < 4; ++k) Op::step(acc[k], v[k], w);
		}
	T* o = a.out + y * a.orow + x;
#pragma unroll
	for (int k = 0; k < 4; ++k)
		if (x + 32 * k < a.w) o[32 * k] = Op::end(acc[k], a.c);
}

// ---- host: does memory m read (or write) element (y + base, x + base) of a
// (size2, size3) image, moved by (sy, sx) per window element?
inline bool image_map(const umi_mem_plan& m, bool loop, int* sy, int* sx) {
	for (int k = 0; k < 4; ++k)
		for (int d = 0; d < 4; ++d) {
			const bool diag = k == d && k >= 2;
			if (m.pcoef[k][d] != (diag ? 1 : 0)) return false;
			if (!diag && m.acoef[k][d] != 0) return false;
			if (diag && !loop && m.acoef[k][d] != 0) return false;
		}
	if (m.base[0] != 0 || m.base[1] != 0) return false;
	if (sy) *sy = m.acoef[2][2];
	if (sx) *sx = m.acoef[3][3];
	return true;
}

template <class Op, int KX>
umi_status launch_kx(const Args<Op>& a, dim3 grid, size_t smem, cudaStream_t st) {
	auto kern = window_kernel<Op, KX>;
	UMI_TRY(umi::allow_shared(kern, smem));
	kern<<<grid, NT, smem, st>>>(a);
	return UMI_OK;
}

// An instance for every odd number of window columns up to 7 (15 with weights),
// the widths of centred windows; one loop for the others.  (Two float passes of
// 9 and 15 taps, 2160 x 3840: 35 and 41 us with the loop, 33 and 38.5 so.)
template <class Op, int KX>
umi_status launch_columns(const Args<Op>& a, dim3 grid, size_t smem, cudaStream_t st) {
	if (a.kx == KX) return launch_kx<Op, KX>(a, grid, smem, st);
	if constexpr (KX + 2 <= (Op::kWeights ? 15 : 7)) return launch_columns<Op, KX + 2>(a, grid, smem, st);
	return launch_kx<Op, 0>(a, grid, smem, st);
}

constexpr int kMaxTile = 96 * 1024;  // bytes of shared memory for the staged tile

// Runs the plan if it is a window operator of `Op` (memories: [centre,] image
// [, weights], output); *done says whether it did.  What is left to the
// generic kernel: other P or A spaces, a window in several accumulation
// blocks (another order), outer image dimensions, images whose rows or elements
// are not contiguous, indices beyond 32 bits.
//
// 1080p on a GB300, us per launch under ncu (cold caches), generic kernel ->
// window kernel: census 5x5 51.5 -> 12.9, 3x3 37.8 -> 9.8; dilation 3x3 35.2
// -> 7.3; erosion 7x7 70.4 -> 10.3; 13 float taps across 51.7 -> 10.2, down
// 102 -> 9.0; strided kernel: four corners of a box sum 51.2 -> 8.3.
template <class Op>
umi_status window_launch(const umi_plan& plan, const UMI::gpu_detail::LinearMaps& lm, const void* const* in,
                         const void* pad, void* out, const typename Op::C& c, cudaStream_t st, bool* done) {
	using T = typename Op::T;
	*done = false;
	if (!lm.fit32 || !lm.idx32 || plan.ptotal[0] != 1 || plan.ptotal[1] != 1 || plan.atotal[0] != 1 ||
	    plan.atotal[1] != 1 || plan.n_ablock != 1)
		return UMI_OK;
	constexpr int CI = 0, II = Op::kCentre ? 1 : 0, WI = II + 1, OI = II + 1 + (Op::kWeights ? 1 : 0);
	Args<Op> a;
	std::memset(&a, 0, sizeof(a));
	a.h = plan.ptotal[2]; a.w = plan.ptotal[3];
	a.ky = plan.atotal[2]; a.kx = plan.atotal[3];
	auto image = [&](int m, Image<T>* im) {
		const umi_mem_plan& mp = plan.mem[m];
		if (mp.size[0] < 1 || mp.size[1] < 1 || mp.size[2] < 1 || mp.size[3] < 1) return false;
		// a plan's row strides may be the caller's own (rows of a pitched image)
		if (mp.rowstride[3] != 1 || mp.rowstride[2] != mp.size[3]) return false;
		im->p = static_cast<const T*>(in[m]);
		im->h = mp.size[2]; im->w = mp.size[3];
		im->oy = mp.base[2]; im->ox = mp.base[3];
		im->pad_y = mp.pad_mask >> 2 & 1; im->pad_x = mp.pad_mask >> 3 & 1;
		if (pad) std::memcpy(&im->pad, static_cast<const char*>(pad) + 4 * m, sizeof(T));
		return true;
	};
	if (!image_map(plan.mem[II], true, &a.sy, &a.sx) || !image(II, &a.img)) return UMI_OK;
	if (a.ky == 1) a.sy = 1;  // no step is taken
	if (a.kx == 1) a.sx = 1;
	if (Op::kCentre && (!image_map(plan.mem[CI], false, nullptr, nullptr) || !image(CI, &a.centre))) return UMI_OK;
	a.cy = -1;
	if (Op::kCentre) {
		const int cy = a.centre.oy - a.img.oy, cx = a.centre.ox - a.img.ox;
		if (a.centre.p == a.img.p && a.centre.h == a.img.h && a.centre.w == a.img.w && a.centre.pad_y == a.img.pad_y &&
		    a.centre.pad_x == a.img.pad_x && std::memcmp(&a.centre.pad, &a.img.pad, sizeof(T)) == 0 && cy >= 0 && cy < a.ky &&
		    cx >= 0 && cx < a.kx) {
			a.cy = cy;
			a.cx = cx;
		}
	}
	if (Op::kWeights) {  // one value per window element, every element inside the weights' extent
		const umi_mem_plan& mp = plan.mem[WI];
		for (int k = 0; k < 4; ++k) {
			for (int d = 0; d < 4; ++d)
				if (mp.pcoef[k][d] != 0) return UMI_OK;
			if (mp.base[k] + lm.alo[WI][k] < 0 || mp.base[k] + lm.ahi[WI][k] > mp.size[k] - 1) return UMI_OK;
		}
		a.wts = static_cast<const T*>(in[WI]) + lm.lin[WI];
		a.wsy = (int)lm.astr[WI][2];
		a.wsx = (int)lm.astr[WI][3];
	}
	for (int d = 0; d < 4; ++d)  // the output row is contiguous along x
		if (d != 2 && lm.pstr[OI][d] != (d == 3 ? 1 : 0) && plan.ptotal[d] > 1) return UMI_OK;
	a.out = static_cast<T*>(out) + lm.lin[OI];
	a.orow = lm.pstr[OI][2];
	a.vec = umi::aligned(a.out, 16) && a.orow % 4 == 0;
	a.c = c;
	a.tw = TX + ((a.kx + 3) & ~3);
	const int64_t tile = 4 * ((int64_t)(TY + a.ky - 1) * a.tw + (Op::kWeights ? (int64_t)a.ky * ((a.kx + 3) & ~3) : 0));
	const int64_t gx = umi::ceil_div(a.w, TX);
	if (a.sy == 1 && a.sx == 1 && tile <= kMaxTile && umi::ceil_div(a.h, TY) <= 65535) {
		const dim3 grid((unsigned)gx, (unsigned)umi::ceil_div(a.h, TY));
		UMI_TRY((launch_columns<Op, 1>(a, grid, (size_t)tile, st)));
	} else if (umi::ceil_div(a.h, NT / 32) <= 65535) {
		strided_kernel<Op><<<dim3((unsigned)gx, (unsigned)umi::ceil_div(a.h, NT / 32)), NT, 0, st>>>(a);
	} else {
		return UMI_OK;
	}
	*done = true;
	return umi::launch_status("window_kernel");
}

}  // namespace umi_window
