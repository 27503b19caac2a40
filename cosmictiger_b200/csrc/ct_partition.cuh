// Warp helpers of the exact two-pointer partitions (tree build and rung sort): a warp holds up to 1,024
// elements as one ballot word a lane.
#pragma once
#include "ct_internal.cuh"

namespace ct {
namespace {

// The first n bits of a lane's word that starts at bit `first`.
__device__ __forceinline__ unsigned first_bits(int n, int first) {
	return first >= n ? 0u : (n - first >= 32 ? 0xffffffffu : (1u << (n - first)) - 1u);
}
__device__ __forceinline__ int lane_scan(int v, int lane) {
	for (int o = 1; o < 32; o <<= 1) {
		const int t = __shfl_up_sync(0xffffffffu, v, o);
		v += lane >= o ? t : 0;
	}
	return v;
}
// Particles of a SUB on the wrong side of the split point, which lies after `before` of its n: those
// before it that are not below the midpoint go to left(rank from the SUB's left, offset), those after
// it that are below to right(rank from its right, offset).
template<class L, class R>
__device__ __forceinline__ void sub_wrong(unsigned mine, int n, int before, int lane, L left, R right) {
	const unsigned bf = first_bits(before, 32 * lane);
	unsigned l = bf & ~mine & first_bits(n, 32 * lane), r = mine & ~bf;
	int k = lane_scan(__popc(l), lane) - __popc(l);
	while (l) {
		left(k++, 32 * lane + __ffs(l) - 1);
		l &= l - 1;
	}
	const int ir = lane_scan(__popc(r), lane);
	k = __shfl_sync(0xffffffffu, ir, 31) - 1 - (ir - __popc(r));
	while (r) {
		right(k--, 32 * lane + __ffs(r) - 1);
		r &= r - 1;
	}
}

}  // namespace
}  // namespace ct
