// What the grouped GEMM kernels share: the search for a tile's problem and the offsets of split dimensions.
#pragma once
#include "common.cuh"

namespace ttc {

// The problem that a tile belongs to: the last one whose tile_start is not above it.  Each round of the
// search reads 32 descriptors at once, one per lane (two rounds of loads up to 1024 problems).
__device__ __forceinline__ int find_desc(const GemmDesc* __restrict__ d, int nd, long long tile) {
  const int lane = threadIdx.x & 31;
  int lo = 0, end = nd;
  while (end - lo > 1) {
    const int step = (end - lo + 31) >> 5, at = lo + lane * step;
    const unsigned in = __ballot_sync(0xffffffffu, at < end && d[at].tile_start <= tile);
    lo += (__popc(in) - 1) * step;
    end = min(end, lo + step);
  }
  return lo;
}

// Offset of index g of a dimension split as g = g0 + n0 g1 with strides s0, s1; one: n0 covers the dimension.
__device__ __forceinline__ long long split_off(int g, int n0, bool one, long long s0, long long s1) {
  if (one) return (long long)g * s0;
  const int q = g / n0;
  return (long long)(g - q * n0) * s0 + (long long)q * s1;
}

}  // namespace ttc
