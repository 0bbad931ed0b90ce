// Kernels of the motion-proposal network's training pass (learned_me.cu):
// convolution forward, weight gradient and head, on fp32 planar activations
// (C, H, W) with W a multiple of 4.  (The data gradient: menet_parts.cu.)
//
// The FP32 pipe bounds the pass (9.6 GFLOP per 32 -> 32 layer and direction at
// 4K, 0.12 ms at its peak): the kernels keep it fed with packed fp32 pairs
// (fma.rn.f32x2, two independent IEEE FMAs per instruction, so half the issue
// slots) on register tiles of 64-72 accumulators per thread.  Measured at
// 2160 x 3840 on a GB300, before -> now (before: scalar FMAs, 9-10 shared
// loads per tap of two pixels or one, one partial row per 4 x 32 pixels):
// forward 0.39-0.45 -> 0.21-0.23 ms a layer (FMA pipe 60-64 % busy, the rest is
// the last wave of tiles and the barriers), weight gradient 0.92-1.07 ->
// 0.22-0.24 ms (53-58 %) and its reduction 0.37 -> 0.008 ms, head 0.64 -> 0.05
// ms; forward + backward 7.5 -> 1.69 ms, the data gradient's part of it on the
// tensor cores (2.15 with it on this pipe).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace menet_train {

constexpr int CH = 32;
constexpr int NT = 256;
constexpr int HEADF = CH * 16;
constexpr int PARTS = 304;       // partial sums of the gradients: two CTAs per SM
constexpr int HEAD_PARTS = 912;  // the head's: six smaller CTAs per SM

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
	uint64_t d;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
	return d;
}
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
	uint64_t d;
	asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
	return d;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
	float2 f;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
	return f;
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {  // zero fill when not valid
	const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// 16 bytes of shared memory, kept in program order (a plain load would be
// hoisted over the unrolled loops and spill the accumulators)
__device__ __forceinline__ ulonglong2 lds16(unsigned addr) {
	ulonglong2 v;
	asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
	return v;
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() {
	asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Staged row of a 32-column strip: columns x0 - HALO .. x0 + 31 + HALO, whole
// 16-byte pieces; the row stride is an odd number of pieces, so 16-byte loads
// of eight rows (or of two rows by four lanes) fall into distinct banks.
template <int DIL> struct Strip {
	static_assert(DIL % 2 == 0, "pixel pairs of every tap start at an even column");
	static constexpr int HALO = DIL < 4 ? 4 : DIL;
	static constexpr int TW = 32 + 2 * HALO, Q = TW / 4;
	static constexpr int TWP = TW + (Q % 2 ? 0 : 4);
	static constexpr int TAP0 = (HALO - DIL) / 2;  // pair of tap column 0; the next ones DIL / 2 pairs on
};

// ---- weights rounded to bf16.  Forward in fp32, fwd[ci][tap][co], after layer
// 0 every value twice (the constant operand of fma2); for the data gradient of
// the 32 -> 32 layers transposed and flipped, as K-major bf16 matrices
// bwd[ci][8 - tap][co] (menet_parts.cu).
struct Pack {
	const float* w[4];
	float* fwd[4];
	__nv_bfloat16* bwd[4];
};
__global__ void pack_weights_kernel(const Pack p, int first) {
	const int l = first + blockIdx.y, cin = l == 0 ? 2 : CH;
	const float* w = l == 0 ? p.w[0] : l == 1 ? p.w[1] : l == 2 ? p.w[2] : p.w[3];
	float* fwd = l == 0 ? p.fwd[0] : l == 1 ? p.fwd[1] : l == 2 ? p.fwd[2] : p.fwd[3];
	__nv_bfloat16* bwd = l == 1 ? p.bwd[1] : l == 2 ? p.bwd[2] : p.bwd[3];
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < CH * cin * 9; i += gridDim.x * blockDim.x) {
		const int co = i / (cin * 9), r = i - co * cin * 9, ci = r / 9, tap = r - ci * 9;
		const __nv_bfloat16 b = __float2bfloat16_rn(w[i]);
		const float v = __bfloat162float(b);
		if (l == 0) {
			fwd[r * CH + co] = v;
		} else {
			reinterpret_cast<float2*>(fwd)[r * CH + co] = make_float2(v, v);
			bwd[(ci * 9 + 8 - tap) * CH + co] = b;
		}
	}
}

// ---- layer 1 (2 -> 32 channels, dilation 1): bound by its 66 MB of output
// at 4K.  A thread computes 4 adjacent pixels x 32 channels, eight channels
// (four pairs) at a time, from a 3 x 6 window per input channel.  Each output
// sums bias, then the 18 products in (ci, tap) order.
__global__ void __launch_bounds__(NT) conv_first_kernel(const float* __restrict__ x0, const float* __restrict__ w,
                                                        const float* __restrict__ bias, float* __restrict__ out, int H,
                                                        int W) {
	__shared__ __align__(16) float ws[18 * CH];
	__shared__ __align__(16) float bs[CH];
	for (int i = threadIdx.x; i < 18 * CH; i += NT) ws[i] = w[i];
	if (threadIdx.x < CH) bs[threadIdx.x] = bias[threadIdx.x];
	__syncthreads();
	const int P = H * W, gx = W >> 2, g = blockIdx.x * NT + threadIdx.x;
	if (g >= H * gx) return;
	const int y = g / gx, x = (g - y * gx) * 4;
	float in[2][3][6];
#pragma unroll
	for (int ci = 0; ci < 2; ++ci)
#pragma unroll
		for (int r = 0; r < 3; ++r) {
			const int yy = y + r - 1;
#pragma unroll
			for (int c = 0; c < 6; ++c) in[ci][r][c] = 0.0f;
			if (yy >= 0 && yy < H) {
				const float* row = x0 + (size_t)ci * P + (size_t)yy * W + x;
				const float4 m = __ldg(reinterpret_cast<const float4*>(row));
				if (x > 0) in[ci][r][0] = __ldg(row - 1);
				in[ci][r][1] = m.x; in[ci][r][2] = m.y; in[ci][r][3] = m.z; in[ci][r][4] = m.w;
				if (x + 4 < W) in[ci][r][5] = __ldg(row + 4);
			}
		}
#pragma unroll 1
	for (int q = 0; q < 4; ++q) {
		uint64_t acc[4][4];  // [channel pair][pixel]
		const ulonglong2 ba = *reinterpret_cast<const ulonglong2*>(bs + 8 * q);
		const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(bs + 8 * q + 4);
#pragma unroll
		for (int px = 0; px < 4; ++px) { acc[0][px] = ba.x; acc[1][px] = ba.y; acc[2][px] = bb.x; acc[3][px] = bb.y; }
#pragma unroll
		for (int k = 0; k < 18; ++k) {
			const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(ws + k * CH + 8 * q);
			const ulonglong2 wb = *reinterpret_cast<const ulonglong2*>(ws + k * CH + 8 * q + 4);
#pragma unroll
			for (int px = 0; px < 4; ++px) {
				const float v = in[k / 9][(k % 9) / 3][px + k % 3];
				const uint64_t vv = pair(v, v);
				acc[0][px] = fma2(wa.x, vv, acc[0][px]);
				acc[1][px] = fma2(wa.y, vv, acc[1][px]);
				acc[2][px] = fma2(wb.x, vv, acc[2][px]);
				acc[3][px] = fma2(wb.y, vv, acc[3][px]);
			}
		}
#pragma unroll
		for (int c = 0; c < 4; ++c) {
			const float2 a = unpair(acc[c][0]), b = unpair(acc[c][1]), d = unpair(acc[c][2]), e = unpair(acc[c][3]);
			float* o = out + (size_t)(8 * q + 2 * c) * P + (size_t)y * W + x;
			*reinterpret_cast<float4*>(o) = make_float4(fmaxf(a.x, 0.f), fmaxf(b.x, 0.f), fmaxf(d.x, 0.f), fmaxf(e.x, 0.f));
			*reinterpret_cast<float4*>(o + P) =
				make_float4(fmaxf(a.y, 0.f), fmaxf(b.y, 0.f), fmaxf(d.y, 0.f), fmaxf(e.y, 0.f));
		}
	}
}

// ---- layers 2-4, forward (32 -> 32 channels).
//   out[co][p] = relu( bias[co] + sum_{ci,tap} w[ci][tap][co] in[ci][p + DIL off(tap)] ),
// zero outside the image.  CTA: 32 x 16 pixels x 32 channels; a warp owns 8 channels and 8
// rows, a thread 8 adjacent pixels (four pairs) x 8 channels.  Per input
// channel and tap row it reads 4-6 16-byte pieces of its pixel row and 12 of
// doubled weights (one address per warp) for 96 fma2.  Two input channels per
// stage, three stages in flight (cp.async; zero fill outside the image).
// Every output sums bias, then (ci, tap) in order, one FMA each.
template <int DIL> struct ConvTile : Strip<DIL> {
	static constexpr int TH = 16 + 2 * DIL, CPS = 2, STAGES = 3;
	static constexpr int ACT = CPS * TH * Strip<DIL>::TWP, WST = CPS * 9 * CH * 2;
	static constexpr size_t smem = sizeof(float) * STAGES * (ACT + WST);
};

template <int DIL>
__global__ void __launch_bounds__(NT, 2) conv_kernel(const float* __restrict__ in, const float* __restrict__ wdup,
                                                     const float* __restrict__ bias, float* __restrict__ out, int H,
                                                     int W) {
	using T = ConvTile<DIL>;
	constexpr int TH = T::TH, TWP = T::TWP, Q = T::Q, STG = T::ACT + T::WST;
	constexpr int NQ = (T::TAP0 * 2 + 2 * DIL + 8 + 3) / 4;  // pieces of a row a thread reads
	extern __shared__ __align__(16) float sm[];
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int cg = warp >> 1, row = (warp & 1) * 8 + (lane >> 2), xq = (lane & 3) * 8;
	const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 16, P = H * W;
	auto stage = [&](int s) {
		if (s < CH / T::CPS) {
			float* a = sm + (s % T::STAGES) * STG;
			const float* src = in + (size_t)(s * T::CPS) * P;
			for (int i = tid; i < T::CPS * TH * Q; i += NT) {
				const int c = i / (TH * Q), r = i - c * (TH * Q), sy = r / Q, q = r - sy * Q;
				const int gy = y0 - DIL + sy, gx = x0 - T::HALO + 4 * q;
				const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
				copy16(a + (c * TH + sy) * TWP + 4 * q, ok ? src + (size_t)c * P + (size_t)gy * W + gx : in, ok);
			}
			const float* wsrc = wdup + (size_t)s * T::WST;
			for (int i = tid; i < T::WST / 4; i += NT) copy16(a + T::ACT + 4 * i, wsrc + 4 * i, true);
		}
		copy_commit();
	};
	uint64_t acc[8][4];  // [channel][pixel pair]
#pragma unroll
	for (int c = 0; c < 8; ++c) {
		const float b = __ldg(bias + 8 * cg + c);
#pragma unroll
		for (int p = 0; p < 4; ++p) acc[c][p] = pair(b, b);
	}
	stage(0);
	stage(1);
	for (int s = 0; s < CH / T::CPS; ++s) {
		copy_wait<1>();
		__syncthreads();
		stage(s + 2);  // the buffer of stage s - 1, which every thread has left
		const float* a = sm + (s % T::STAGES) * STG;
#pragma unroll 1
		for (int c = 0; c < T::CPS; ++c) {
			const float* w = a + T::ACT + (c * 9 * CH + 8 * cg) * 2;
#pragma unroll
			for (int ty = 0; ty < 3; ++ty) {
				uint64_t v[2 * NQ];
#pragma unroll
				for (int q = 0; q < NQ; ++q) {
					const ulonglong2 t =
						*reinterpret_cast<const ulonglong2*>(a + (c * TH + row + ty * DIL) * TWP + xq + 4 * q);
					v[2 * q] = t.x;
					v[2 * q + 1] = t.y;
				}
#pragma unroll
				for (int tx = 0; tx < 3; ++tx)
#pragma unroll
					for (int k = 0; k < 4; ++k) {
						const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(w + (ty * 3 + tx) * CH * 2 + 4 * k);
#pragma unroll
						for (int p = 0; p < 4; ++p) {
							const uint64_t x = v[T::TAP0 + tx * (DIL / 2) + p];
							acc[2 * k][p] = fma2(wv.x, x, acc[2 * k][p]);
							acc[2 * k + 1][p] = fma2(wv.y, x, acc[2 * k + 1][p]);
						}
					}
			}
		}
	}
	const int y = y0 + row;
	if (y >= H) return;
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		const int x = x0 + xq + 4 * h;
		if (x >= W) break;
#pragma unroll
		for (int c = 0; c < 8; ++c) {
			const float2 l = unpair(acc[c][2 * h]), r = unpair(acc[c][2 * h + 1]);
			const size_t p = (size_t)(8 * cg + c) * P + (size_t)y * W + x;
			const float4 o = make_float4(fmaxf(l.x, 0.f), fmaxf(l.y, 0.f), fmaxf(r.x, 0.f), fmaxf(r.y, 0.f));
			*reinterpret_cast<float4*>(out + p) = o;
		}
	}
}

// ---- the order in which the weight-gradient CTAs walk the image: strips of
// 32 columns; inside a strip the rows of one dilation class, y = c, c + DIL,
// c + 2 DIL, ..., class after class, so that consecutive rows share two of
// their three tap rows.  Row i of a strip, and its successor.
struct RowWalk {
	int strip, y;
	__host__ __device__ static RowWalk at(int unit, int H, int dil) {
		RowWalk w;
		w.strip = unit / H;
		int i = unit - w.strip * H, c = 0;
		for (;;) {
			const int n = (H - c + dil - 1) / dil;  // rows of class c
			if (i < n) break;
			i -= n;
			++c;
		}
		w.y = c + i * dil;
		return w;
	}
	// moves on; true when the next row continues the run (y + dil of the same strip)
	__host__ __device__ bool next(int H, int dil) {
		if (y + dil < H) {
			y += dil;
			return true;
		}
		const int c = y % dil + 1;
		if (c < dil && c < H) {
			y = c;
		} else {
			y = 0;
			++strip;
		}
		return false;
	}
};

// ---- weight gradient of layers 2-4:
//   part[cta][co][ci][tap] = sum over the CTA's pixels of dpre[co][p] in[ci][p + DIL off(tap)],
// then the bias part sum_p dpre[co][p].  Each CTA walks a contiguous piece of
// the row order above and keeps its sums in registers: warp = 4 output
// channels, lane = input channel, a thread 4 x 9 sums of even and of odd
// pixels (72 accumulators).  Shared memory holds a ring of four input rows
// (all channels) and two gradient rows; the next row arrives (cp.async) while
// one is used.  Per four pixels and tap row a thread reads one piece of its
// input row (the taps of a row overlap) and four of gradients (one address
// per warp) for 24 fma2.
template <int DIL> struct WgradTile : Strip<DIL> {
	static constexpr int ROW = CH * Strip<DIL>::TWP;  // floats of a staged input row
	static constexpr size_t smem = sizeof(float) * (4 * ROW + 2 * CH * 32);
};

template <int DIL>
__global__ void __launch_bounds__(NT, 2) wgrad_kernel(const float* __restrict__ in, const float* __restrict__ dpre,
                                                      float* __restrict__ part, int H, int W, int units, int per) {
	using T = WgradTile<DIL>;
	constexpr int TWP = T::TWP, Q = T::Q, NP = (2 * T::TAP0 + 2 * DIL + 4 + 3) / 4;
	static_assert(8 + NP - 1 <= Q, "pieces of a staged row");
	extern __shared__ __align__(16) float sm[];
	float* xs = sm;               // [4][CH][TWP]
	float* ds = sm + 4 * T::ROW;  // [2][CH][32]
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, P = H * W;
	const int u0 = blockIdx.x * per, u1 = min(units, u0 + per);
	const int dc = tid >> 3, dq = tid & 7;  // the gradient piece this thread stages
	auto load_row = [&](int slot, int strip, int y) {
		const bool rok = y >= 0 && y < H;
#pragma unroll 1
		for (int i = tid; i < CH * Q; i += NT) {
			const int c = i / Q, q = i - c * Q, gx = strip * 32 - T::HALO + 4 * q;
			const bool ok = rok && gx >= 0 && gx < W;
			copy16(xs + slot * T::ROW + c * TWP + 4 * q, ok ? in + (size_t)c * P + (size_t)y * W + gx : in, ok);
		}
	};
	auto load_d = [&](const RowWalk& w) {
		const int gx = w.strip * 32 + 4 * dq;
		return gx < W ? __ldg(reinterpret_cast<const float4*>(dpre + (size_t)dc * P + (size_t)w.y * W + gx))
		              : make_float4(0.f, 0.f, 0.f, 0.f);
	};
	uint64_t acc[4][9];
#pragma unroll
	for (int c = 0; c < 4; ++c)
#pragma unroll
		for (int t = 0; t < 9; ++t) acc[c][t] = 0;
	float4 bsum = make_float4(0.f, 0.f, 0.f, 0.f);
	if (u0 < u1) {
		RowWalk w = RowWalk::at(u0, H, DIL);
		float4 dv = load_d(w);
		bool fresh = true;
		int b = 0;  // slots b, b + 1, b + 2 (mod 4): rows y - DIL, y, y + DIL
		for (int u = u0; u < u1; ++u) {
			if (fresh)
#pragma unroll 1
				for (int k = 0; k < 3; ++k) load_row((b + k) & 3, w.strip, w.y + (k - 1) * DIL);
			copy_commit();
			copy_wait<0>();
			float* d = ds + (u & 1) * (CH * 32);
			*reinterpret_cast<float4*>(d + dc * 32 + 4 * dq) = dv;
			bsum.x += dv.x; bsum.y += dv.y; bsum.z += dv.z; bsum.w += dv.w;
			__syncthreads();
			RowWalk nw = w;
			const bool cont = nw.next(H, DIL);
			if (u + 1 < u1) {
				if (cont) load_row((b + 3) & 3, nw.strip, nw.y + DIL);  // the slot of row y - 2 DIL, left by every thread
				dv = load_d(nw);
			}
#pragma unroll
			for (int ty = 0; ty < 3; ++ty) {
				const unsigned xr = (unsigned)__cvta_generic_to_shared(xs + ((b + ty) & 3) * T::ROW + lane * TWP);
				const unsigned dr = (unsigned)__cvta_generic_to_shared(d + warp * 4 * 32);
				// pieces q .. q + NP - 1 of the row serve pixels 4 q .. 4 q + 3 of all
				// three tap columns; two rolled halves of 16 pixels keep the
				// window's registers few (fully unrolled it spills)
				uint64_t xv[2 * (4 + NP - 1)];
				auto piece = [&](int at, int q) {
					const ulonglong2 t = lds16(xr + 16 * q);
					xv[2 * at] = t.x;
					xv[2 * at + 1] = t.y;
				};
#pragma unroll
				for (int q = 0; q < NP - 1; ++q) piece(q, q);
#pragma unroll 1
				for (int h = 0; h < 2; ++h) {
#pragma unroll
					for (int q = 0; q < 4; ++q) {
						piece(q + NP - 1, 4 * h + q + NP - 1);
#pragma unroll
						for (int c = 0; c < 4; ++c) {
							const ulonglong2 g = lds16(dr + 4 * (c * 32 + 16 * h + 4 * q));
#pragma unroll
							for (int tx = 0; tx < 3; ++tx) {
								const int k = T::TAP0 + tx * (DIL / 2) + 2 * q;
								acc[c][ty * 3 + tx] = fma2(g.x, xv[k], acc[c][ty * 3 + tx]);
								acc[c][ty * 3 + tx] = fma2(g.y, xv[k + 1], acc[c][ty * 3 + tx]);
							}
						}
					}
#pragma unroll
					for (int i = 0; i < 2 * (NP - 1); ++i) xv[i] = xv[8 + i];
				}
			}
			if (u + 1 < u1 && !cont) __syncthreads();  // the next run's rows overwrite this one's
			fresh = !cont;
			b = (b + 1) & 3;
			w = nw;
		}
	}
	float* dst = part + (size_t)blockIdx.x * (CH * CH * 9 + CH);
#pragma unroll
	for (int c = 0; c < 4; ++c)
#pragma unroll
		for (int t = 0; t < 9; ++t) {
			const float2 s = unpair(acc[c][t]);
			dst[((4 * warp + c) * CH + lane) * 9 + t] = s.x + s.y;
		}
	float s = (bsum.x + bsum.y) + (bsum.z + bsum.w);
#pragma unroll
	for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	if (dq == 0) dst[CH * CH * 9 + dc] = s;
}

// Weight gradient of layer 1 (2 input channels, dilation 1): bound by reading
// the 66 MB of gradients once.  Warp = 4 output channels, lane = column of a
// 32-column strip; a thread walks down its column with the 3 x 3 windows of
// both input channels in registers and 72 sums, reduced over the lanes at the
// end.
__global__ void __launch_bounds__(NT, 2) wgrad_first_kernel(const float* __restrict__ in,
                                                            const float* __restrict__ dpre, float* __restrict__ part,
                                                            int H, int W, int units, int per) {
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, P = H * W;
	const int u0 = blockIdx.x * per, u1 = min(units, u0 + per);
	float acc[4][18], bacc[4];
#pragma unroll
	for (int c = 0; c < 4; ++c) {
		bacc[c] = 0.0f;
#pragma unroll
		for (int t = 0; t < 18; ++t) acc[c][t] = 0.0f;
	}
	auto load_x = [&](int strip, int y, float (&v)[2][3]) {
		const int x = strip * 32 + lane;
#pragma unroll
		for (int ci = 0; ci < 2; ++ci)
#pragma unroll
			for (int k = 0; k < 3; ++k) {
				const int xx = x + k - 1;
				v[ci][k] = y >= 0 && y < H && xx >= 0 && xx < W ? __ldg(in + (size_t)ci * P + (size_t)y * W + xx) : 0.0f;
			}
	};
	auto load_d = [&](int strip, int y, float (&v)[4]) {
		const int x = strip * 32 + lane;
#pragma unroll
		for (int c = 0; c < 4; ++c)
			v[c] = y < H && x < W ? __ldg(dpre + (size_t)(4 * warp + c) * P + (size_t)y * W + x) : 0.0f;
	};
	for (int u = u0; u < u1;) {  // one piece of a strip: rows y .. ye - 1
		const int strip = u / H, y0 = u - strip * H, ye = min(H, y0 + u1 - u);
		float r0[2][3], r1[2][3];
		load_x(strip, y0 - 1, r0);
		load_x(strip, y0, r1);
#pragma unroll 2
		for (int y = y0; y < ye; ++y) {
			float r2[2][3], d[4];
			load_x(strip, y + 1, r2);
			load_d(strip, y, d);
#pragma unroll
			for (int c = 0; c < 4; ++c) {
				bacc[c] += d[c];
#pragma unroll
				for (int ci = 0; ci < 2; ++ci)
#pragma unroll
					for (int k = 0; k < 3; ++k) {
						acc[c][ci * 9 + k] = fmaf(d[c], r0[ci][k], acc[c][ci * 9 + k]);
						acc[c][ci * 9 + 3 + k] = fmaf(d[c], r1[ci][k], acc[c][ci * 9 + 3 + k]);
						acc[c][ci * 9 + 6 + k] = fmaf(d[c], r2[ci][k], acc[c][ci * 9 + 6 + k]);
					}
			}
#pragma unroll
			for (int ci = 0; ci < 2; ++ci)
#pragma unroll
				for (int k = 0; k < 3; ++k) {
					r0[ci][k] = r1[ci][k];
					r1[ci][k] = r2[ci][k];
				}
		}
		u += ye - y0;
	}
	float* dst = part + (size_t)blockIdx.x * (CH * 18 + CH);
#pragma unroll
	for (int c = 0; c < 4; ++c) {
#pragma unroll
		for (int t = 0; t < 19; ++t) {
			float s = t < 18 ? acc[c][t < 18 ? t : 0] : bacc[c];
#pragma unroll
			for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
			if (lane == 0) dst[t < 18 ? (4 * warp + c) * 18 + t : CH * 18 + 4 * warp + c] = s;
		}
	}
}

// out[j] = sum over the n rows of the row-major (n, m) array, j < m - (extra
// != null), in a fixed order; the last column goes to *extra when given.  A
// CTA takes 32 columns, its 8 warps every 8th row each.  Where a data gradient
// that the rows come from is not complete (bits in *err) the sums are NaN, and
// the bits are added to *report when given.
__global__ void __launch_bounds__(NT) reduce_rows_kernel(const float* __restrict__ part, float* __restrict__ out,
                                                         float* __restrict__ extra, int n, int m, int cols,
                                                         const int32_t* __restrict__ err, int32_t* __restrict__ report) {
	__shared__ float red[8][32];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, j = blockIdx.x * 32 + lane;
	float s[4] = {0.f, 0.f, 0.f, 0.f};
	if (j < m) {
		int i = warp;
		for (; i + 24 < n; i += 32)
#pragma unroll
			for (int k = 0; k < 4; ++k) s[k] += __ldg(part + (size_t)(i + 8 * k) * m + j);
		for (int k = 0; i < n; i += 8, ++k) s[k] += __ldg(part + (size_t)i * m + j);
	}
	red[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
	__syncthreads();
	if (warp == 0 && j < m) {
		float t = 0.0f;
#pragma unroll
		for (int k = 0; k < 8; ++k) t += red[k][lane];
		const int32_t bits = *err;
		if (bits) t = __int_as_float(0x7fffffff);
		if (bits && report && j == 0) atomicOr(report, bits);
		if (j < cols) out[j] = t;
		else if (extra) *extra = t;
	}
}

// ---- head, forward: pred[blk][j] = bh[j] + sum_f wh[j][f] feature_f.  Bound
// by reading the activations once (66 MB at 4K): a CTA takes 64 blocks of a
// block row, warp = one cell row of 32 of them, lane = block, so every load is
// 512 contiguous bytes.
__global__ void __launch_bounds__(NT) head_fwd_kernel(const float* __restrict__ a4, const float* __restrict__ wh,
                                                      const float* __restrict__ bh, float* __restrict__ pred, int H4,
                                                      int W4, int nbx) {
	__shared__ __align__(16) float ws[2 * HEADF];  // [j][c][cell row][cell]
	__shared__ float red[4][64][2];
	for (int i = threadIdx.x; i < 2 * HEADF; i += NT) ws[i] = __bfloat162float(__float2bfloat16_rn(wh[i]));
	__syncthreads();
	const int i = threadIdx.x >> 6, b = threadIdx.x & 63, bx = blockIdx.x * 64 + b, by = blockIdx.y;
	const size_t P = (size_t)H4 * W4;
	float s0 = 0.0f, s1 = 0.0f;
	if (bx < nbx) {
		const float4* src = reinterpret_cast<const float4*>(a4 + (size_t)(4 * by + i) * W4 + 4 * bx);
#pragma unroll 8
		for (int c = 0; c < CH; ++c) {
			const float4 v = __ldg(src + c * (P / 4));
			const float4 w0 = *reinterpret_cast<const float4*>(ws + c * 16 + i * 4);
			const float4 w1 = *reinterpret_cast<const float4*>(ws + HEADF + c * 16 + i * 4);
			s0 = fmaf(w0.x, v.x, s0); s0 = fmaf(w0.y, v.y, s0); s0 = fmaf(w0.z, v.z, s0); s0 = fmaf(w0.w, v.w, s0);
			s1 = fmaf(w1.x, v.x, s1); s1 = fmaf(w1.y, v.y, s1); s1 = fmaf(w1.z, v.z, s1); s1 = fmaf(w1.w, v.w, s1);
		}
	}
	red[i][b][0] = s0;
	red[i][b][1] = s1;
	__syncthreads();
	if (threadIdx.x < 128) {
		const int k = threadIdx.x >> 1, j = threadIdx.x & 1, x = blockIdx.x * 64 + k;
		if (x < nbx)
			pred[2 * ((size_t)by * nbx + x) + j] = ((red[0][k][j] + red[1][k][j]) + (red[2][k][j] + red[3][k][j])) + bh[j];
	}
}

// ---- head, backward: smooth-L1 loss against target / 16, dpre4 (masked by
// a4 > 0) and per-CTA partials [dWh (2 x 512), dbh (2), loss].  Bound by
// reading and writing one activation array.  A CTA walks tiles of 8 blocks
// of a block row: the tile is read once (128-byte rows), kept in shared
// memory for the weight gradient (thread = two head features), and the
// partials stay in registers until the end.
__global__ void __launch_bounds__(NT) head_bwd_kernel(const float* __restrict__ a4, const float* __restrict__ wh,
                                                      const float* __restrict__ pred, const int32_t* __restrict__ target,
                                                      int tstride, float* __restrict__ dpre4, float* __restrict__ part,
                                                      int H4, int W4, int nbx, int nblk, int tiles_x, int tiles,
                                                      int32_t* __restrict__ err) {
	constexpr int RS = 36, CS = 4 * RS;  // row and channel strides of the tile: 16-byte reads and feature reads spread over the banks
	__shared__ __align__(16) float ws[2 * HEADF];
	__shared__ __align__(16) float tile[CH * CS];
	__shared__ float2 sg[8];
	__shared__ float sl[8];
	const int tid = threadIdx.x;
	if (blockIdx.x == 0 && tid == 0) *err = 0;  // the data gradients' error word
	for (int i = tid; i < 2 * HEADF; i += NT) ws[i] = __bfloat162float(__float2bfloat16_rn(wh[i]));
	const float inv = 1.0f / (float)nblk;
	const size_t P = (size_t)H4 * W4;
	float dw[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, b0 = 0.0f, b1 = 0.0f, loss = 0.0f;
	for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
		const int by = t / tiles_x, bx0 = (t - by * tiles_x) * 8;
		float4 v[4];
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			const int i = tid + NT * k, q = i & 7, r = (i >> 3) & 3, c = i >> 5;
			v[k] = bx0 + q < nbx ? __ldg(reinterpret_cast<const float4*>(a4 + c * P + (size_t)(4 * by + r) * W4 + 4 * (bx0 + q)))
			                     : make_float4(0.f, 0.f, 0.f, 0.f);
		}
		if (tid < 8) {
			float g0 = 0.0f, g1 = 0.0f, l = 0.0f;
			if (bx0 + tid < nbx) {
				const int blk = by * nbx + bx0 + tid;
				const float e0 = pred[2 * blk] - (float)target[(size_t)tstride * blk] * (1.0f / 16.0f);
				const float e1 = pred[2 * blk + 1] - (float)target[(size_t)tstride * blk + 1] * (1.0f / 16.0f);
				l = (fabsf(e0) < 1.0f ? 0.5f * e0 * e0 : fabsf(e0) - 0.5f) +
				    (fabsf(e1) < 1.0f ? 0.5f * e1 * e1 : fabsf(e1) - 0.5f);
				g0 = fminf(fmaxf(e0, -1.0f), 1.0f) * inv;
				g1 = fminf(fmaxf(e1, -1.0f), 1.0f) * inv;
			}
			sg[tid] = make_float2(g0, g1);
			sl[tid] = l * inv;
		}
		__syncthreads();
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			const int i = tid + NT * k, q = i & 7, r = (i >> 3) & 3, c = i >> 5;
			*reinterpret_cast<float4*>(tile + c * CS + r * RS + 4 * q) = v[k];
			const float2 g = sg[q];
			const float4 w0 = *reinterpret_cast<const float4*>(ws + c * 16 + r * 4);
			const float4 w1 = *reinterpret_cast<const float4*>(ws + HEADF + c * 16 + r * 4);
			if (bx0 + q < nbx)
				*reinterpret_cast<float4*>(dpre4 + c * P + (size_t)(4 * by + r) * W4 + 4 * (bx0 + q)) =
					make_float4(v[k].x > 0.0f ? w0.x * g.x + w1.x * g.y : 0.0f, v[k].y > 0.0f ? w0.y * g.x + w1.y * g.y : 0.0f,
					            v[k].z > 0.0f ? w0.z * g.x + w1.z * g.y : 0.0f, v[k].w > 0.0f ? w0.w * g.x + w1.w * g.y : 0.0f);
		}
		__syncthreads();
#pragma unroll
		for (int b = 0; b < 8; ++b) {
			const float2 g = sg[b];
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const int f = tid + NT * h;
				const float a = tile[(f >> 4) * CS + ((f >> 2) & 3) * RS + 4 * b + (f & 3)];
				dw[h][0] = fmaf(g.x, a, dw[h][0]);
				dw[h][1] = fmaf(g.y, a, dw[h][1]);
			}
			if (tid == 0) { b0 += g.x; b1 += g.y; loss += sl[b]; }
		}
		__syncthreads();
	}
	float* dst = part + (size_t)blockIdx.x * (2 * HEADF + 3);
#pragma unroll
	for (int h = 0; h < 2; ++h)
#pragma unroll
		for (int j = 0; j < 2; ++j) dst[j * HEADF + tid + NT * h] = dw[h][j];
	if (tid == 0) {
		dst[2 * HEADF] = b0;
		dst[2 * HEADF + 1] = b1;
		dst[2 * HEADF + 2] = loss;
	}
}

}  // namespace menet_train
