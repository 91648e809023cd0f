// Bounding box of the usable particles of a view, shared by the octree, the
// all-pairs order and the cell list: bb[0..2] receive the ordered bits of the
// minima, bb[3..5] those of the negated maxima (all preset to ~0).
#pragma once
#include <algorithm>
#include <cmath>

#include "amk_internal.cuh"

namespace amk {

constexpr int kBboxThreads = 256;

// A block of four particles per thread up to four blocks per SM, so that the
// loads of a pass are in flight together (one block per SM with a reduction
// per warp into the same six words took 72 us at 1,048,576 particles).
inline unsigned bbox_grid(long n) {
  return static_cast<unsigned>(std::max(1L, std::min(148L * 4, (n + 4 * kBboxThreads - 1) / (4 * kBboxThreads))));
}

// One block's share; `use(i)` tells whether particle i counts.
template <typename Use>
__device__ __forceinline__ void bbox_block(const View& v, Use use, unsigned long long* __restrict__ bb) {
  __shared__ double red[6][kBboxThreads / 32];
  double m[6] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY};
  const long stride = static_cast<long>(gridDim.x) * kBboxThreads;
#pragma unroll 4
  for (long i = blockIdx.x * static_cast<long>(kBboxThreads) + threadIdx.x; i < v.n; i += stride) {
    if (!use(i)) continue;
    const double p[3] = {v.x[i], v.y[i], v.z[i]};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      m[d] = fmin(m[d], p[d]);
      m[3 + d] = fmin(m[3 + d], -p[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m[d] = fmin(m[d], __shfl_xor_sync(0xffffffffu, m[d], o));
    if ((threadIdx.x & 31) == 0) red[d][threadIdx.x >> 5] = m[d];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = red[threadIdx.x][0];
    for (int w = 1; w < kBboxThreads / 32; ++w) r = fmin(r, red[threadIdx.x][w]);
    atomicMin(&bb[threadIdx.x], double_order_bits(r));
  }
}

}  // namespace amk
