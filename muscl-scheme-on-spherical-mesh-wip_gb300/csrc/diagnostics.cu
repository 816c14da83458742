// Device-side diagnostics of a solver state: the per-step sums of
// MUSCL_base.hpp:187-214 (mass, angular momentum, energy, each weighted by
// the face area) and the light curves of physics/adiabatic.hpp:228-333, in
// one pass over the conserved state, so that a caller gets 9 numbers back
// instead of downloading the state.
//
// Light curves: for four observers (x axis, 45 degrees, +z, -z) the sum over
// the faces the observer sees of Pi * cos(alpha) * area.  Visibility and
// cos(alpha) depend on the geometry only and are precomputed on the host with
// the reference's expressions (one plane per observer, 0 where not visible);
// the device evaluates Pi * area once per face and adds its products with the
// observers' cosines by fused multiply-adds.  The sums are reduced in a fixed
// order (per thread, warp and block, then the blocks' partials by the last
// block to finish), so the result is deterministic; it differs from the
// reference's serial sum by the order and by single roundings.  A thread of a
// large mesh adds up to 67 faces in a row (hex(9)); against exact sums of
// random terms on hex(3) .. hex(9) the result is 0.7e-16 .. 1.1e-16 off, as
// a tree of 256-face blocks is (0.3e-16 .. 1.4e-16).
//
// A caller of the light curves waits for them every step, so the pass is one
// launch that leaves its 9 numbers in page-locked host memory (two launches
// and a copy before).  What it takes beyond that is the FP64 pipe's latency,
// 33 ns per dependent instruction (fp64_math.cuh): the 9 sums of a warp are
// reduced together in 16 instructions, each exchange halving the sums a lane
// still carries, instead of 45.  Compiled with -fmad=false like the FP64 step.
#include <cuda_runtime.h>

#include "diagnostics.hpp"
#include "physics_fp64.cuh"

namespace splash {
namespace diag {
namespace {

constexpr int kBlock = 128;
constexpr int kVals = 9;
constexpr int kMaxBlocks = 304;  // 2 per SM: each thread of a large mesh sums several faces

// Sums v[0 .. 16) over the warp: every exchange passes on the half of the
// values that the partner keeps, so lane l ends with the sum of v[l >> 1].
__device__ __forceinline__ double warp_sums(double (&v)[16], int lane) {
#pragma unroll
  for (int o = 16, n = 8; o > 1; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const double got = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[n + k], o);
      v[k] = (up ? v[n + k] : v[k]) + got;
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Sums v over the block; thread k < kVals returns the sum of v[k].
__device__ __forceinline__ double block_sums(double (&v)[16]) {
  __shared__ double sm[kBlock / 32][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s = warp_sums(v, lane);
  __syncthreads();  // the last use of sm
  if ((lane & 1) == 0) sm[warp][lane >> 1] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < kVals) {
    t = sm[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < kBlock / 32; ++w) t = t + sm[w][threadIdx.x];
  }
  return t;
}

__global__ void __launch_bounds__(kBlock) sums_kernel(DiagInput in, double* __restrict__ partial,
                                                      unsigned* __restrict__ done, double* __restrict__ out) {
  double v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = 0.0;
  const size_t fp = in.fpad;
  for (int f = blockIdx.x * kBlock + threadIdx.x; f < in.n_faces; f += gridDim.x * kBlock) {
    double u[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) u[k] = (k < in.dim) ? in.U[k * fp + f] : 0.0;
    const double a = in.area[f];
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = fma(u[k], a, v[k]);
    if (in.light_curves) {
      const f64::D3 r{in.fcn[f], in.fcn[fp + f], in.fcn[2 * fp + f]};
      const double pa = f64::pressure_fc(u, r, in.gam) * a;
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const double c = in.cos_obs[o * fp + f];
        if (f64::bits_of(c) << 1) v[5 + o] = fma(pa, c, v[5 + o]);  // 0 where the observer does not see the face
      }
    }
  }
  const double s = block_sums(v);
  if (threadIdx.x < kVals) {
    partial[(size_t)blockIdx.x * kVals + threadIdx.x] = s;
    __threadfence();
  }
  __shared__ unsigned last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kBlock) {
    const volatile double* p = partial + (size_t)b * kVals;
#pragma unroll
    for (int k = 0; k < kVals; ++k) v[k] = v[k] + p[k];
  }
  const double t = block_sums(v);
  if (threadIdx.x < kVals) out[threadIdx.x] = t;
  if (threadIdx.x == 0) *done = 0u;
}

}  // namespace
}  // namespace diag

int diag_partial_blocks(int n_faces) {
  const int nb = (n_faces + diag::kBlock - 1) / diag::kBlock;
  return nb < diag::kMaxBlocks ? nb : diag::kMaxBlocks;
}

cudaError_t diag_launch(const DiagInput& in, double* partial, unsigned* done, double* out, cudaStream_t st) {
  diag::sums_kernel<<<diag_partial_blocks(in.n_faces), diag::kBlock, 0, st>>>(in, partial, done, out);
  return cudaGetLastError();
}

}  // namespace splash
