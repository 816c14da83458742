// Deterministic block reduction of the per-block partial records of the
// allocation-free dt clip (cfl_noalloc.cu): three maxima (the folds of
// FoldSlot) and five sums.
#pragma once

#include "layout.hpp"

namespace splash {

constexpr int kPartialMaxima = 3;
constexpr int kPartialStride = 8;  // doubles per block partial record

namespace red {

// a merged with b: the first kPartialMaxima values by maximum, the others by sum
__device__ __forceinline__ void merge(double* a, const double* b) {
#pragma unroll
  for (int k = 0; k < kPartialStride; ++k) a[k] = (k < kPartialMaxima) ? fmax(a[k], b[k]) : a[k] + b[k];
}

// Warp + block reduction of the threads' records v; thread 0 of the block
// writes it.  Fixed tree order, so the result is deterministic.
template <int kBlock>
__device__ void block_partials(double (&v)[kPartialStride], double* out) {
  __shared__ double sm[kBlock / 32][kPartialStride];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double b[kPartialStride];
#pragma unroll
    for (int k = 0; k < kPartialStride; ++k) b[k] = __shfl_down_sync(0xffffffffu, v[k], o);
    merge(v, b);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < kPartialStride; ++k) sm[warp][k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBlock / 32; ++w) merge(v, sm[w]);
#pragma unroll
    for (int k = 0; k < kPartialStride; ++k) out[k] = v[k];
  }
}

}  // namespace red
}  // namespace splash
