// Schedule of the rolling-accumulator form of the motion-proposal layers
// (menet_rows_kernel in gemm_tc.cu), kept free of device code so that the
// host tests compile it too.
//
// A CTA walks runs of output rows (rows y, y + d, y + 2d, ... of one
// dilation class and one 128-pixel block).  In a run of `rows` output rows
// whose first is the CTA's row r0, strip m (input row m - 1 of the run,
// m = 0 .. rows + 1) is read by output rows m - dy for the filter rows dy in
// [lo, hi].  The sixteen 32-column accumulators take the CTA's rows in
// descending column order, row r at block roll_slot(r), so the rows
// m - lo, m - lo - 1, ... sit in adjacent blocks from roll_slot(r0 + m - lo)
// up, except where the ring wraps to block 0: the first c1 of the cnt blocks
// come before the wrap, the other cnt - c1 start at block 0.
#pragma once

#ifndef __CUDACC__
#define UMI_ROLL_HD inline
#else
#define UMI_ROLL_HD __host__ __device__ __forceinline__
#endif

namespace umi_roll {

constexpr int kSlots = 16;  // 32-column accumulators: all 512 TMEM columns

template <int SLOTS = kSlots>
UMI_ROLL_HD int slot(int r) {
	return SLOTS - 1 - r % SLOTS;
}

struct Step {
	int lo, hi;  // filter rows reading strip m
	int first;   // accumulator block of output row r0 + m - lo
	int c1;      // blocks before the ring wraps (cnt = hi - lo + 1 in all)
};

template <int SLOTS = kSlots>
UMI_ROLL_HD Step step(int m, int rows, int r0) {
	Step s;
	s.lo = m - rows + 1 > 0 ? m - rows + 1 : 0;
	s.hi = m < 2 ? m : 2;
	s.first = slot<SLOTS>(r0 + m - s.lo);
	const int cnt = s.hi - s.lo + 1;
	s.c1 = cnt < SLOTS - s.first ? cnt : SLOTS - s.first;
	return s;
}

// Row of position pos in a block's order, and the end of its dilation class:
// classes c = y mod d in order, y ascending within a class; classes
// 0 .. rm-1 hold q+1 rows, the others q (q = h / d, rm = h mod d).
UMI_ROLL_HD void row_of(int h, int d, int pos, int& y, int& class_end) {
	const int q = h / d, rm = h - q * d, big = rm * (q + 1);
	if (pos < big) {
		const int c = pos / (q + 1), k = pos - c * (q + 1);
		y = c + k * d;
		class_end = (c + 1) * (q + 1);
	} else {
		const int p2 = pos - big, c = p2 / q, k = p2 - c * q;
		y = rm + c + k * d;
		class_end = big + (c + 1) * q;
	}
}

}  // namespace umi_roll
