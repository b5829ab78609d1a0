// Deterministic block reduction in double: warp shuffles, then the warp totals in warp
// order.  Same launch shape => same bits, run after run.
#pragma once

#include <cuda_runtime.h>

namespace prad {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// all threads of the block must call; all of them get the results
template <int THREADS, int N>
__device__ __forceinline__ void block_sums_d(double (&v)[N]) {
  __shared__ double warp_tot[N][THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = warp_sum_d(v[i]);
  __syncthreads();  // protects warp_tot across back-to-back calls
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (lane == 0) warp_tot[i][w] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    v[i] = 0.0;
#pragma unroll
    for (int k = 0; k < THREADS / 32; ++k) v[i] += warp_tot[i][k];
  }
}
template <int THREADS>
__device__ __forceinline__ double block_sum_d(double x) {
  double v[1] = {x};
  block_sums_d<THREADS>(v);
  return v[0];
}

}  // namespace prad
