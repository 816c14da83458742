// The dt clip of the FP64 step (MUSCL_base.hpp:100-115): folding the faces'
// candidates into the bounds of the next step, and the clip itself.
#pragma once

#include <cstdint>

#include "fp64_math.cuh"
#include "layout.hpp"

namespace splash {
namespace f64 {

// What the folds say of the next step's dt (MUSCL_base.hpp:100-115):
//   CFL bound h0 0.1 / max_vel, max_vel = max(1e-8, sqrt(vel2)),
//   extra dt 0.01 / (|alpha| fric_k sqrt(rate2)), at most 1e20; 1e20 and a flag
//   when some face's is negative (physics/adiabatic.hpp:543-580).
// Where none is, alpha has the sign of every face's rate, so its size serves.
struct DtBounds {
  double max_vel, extra, dt;  // dt: the smaller of the CFL bound and the extra dt
  bool negative;
};
SPLASH_HD DtBounds dt_bounds(double vel2, double rate2, bool negative, const PhysParams& P) {
  DtBounds b;
  b.max_vel = fmax(1e-8, sqrt(vel2));
  const double rate = sqrt(rate2);
  b.negative = negative && !odd_bits(P.alpha);  // an extra dt of -0, or none
  b.extra = 1e20;
  if (!b.negative && rate > 0) b.extra = fmin(1e20, 0.01 / (fabs(P.alpha) * P.fric_k * rate));
  const double cfl = P.h0 * 0.1 / b.max_vel;
  b.dt = (cfl > b.extra) ? b.extra : cfl;
  return b;
}
// dt = min(dt0, 0.1 h0 / max_vel, extra_dt)
SPLASH_HD double clipped_dt(double dt0, double bound) { return less(bound, dt0) ? bound : dt0; }

#if defined(__CUDACC__)
// Folds a warp's candidates (integer maxima: exact in any order) and, in the
// last of n_warps warps to do so, makes the bounds of the next step's dt of
// them and gives the folds a fresh start.  Every lane of the warp calls it.
__device__ __forceinline__ void fold_warp(double vel2, double rate2, bool negative, const DevState& S,
                                          const PhysParams& P, unsigned long long n_warps) {
  unsigned long long v = bits_of(vel2), r = bits_of(rate2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_down_sync(0xffffffffu, v, o);
    const unsigned long long b = __shfl_down_sync(0xffffffffu, r, o);
    v = a > v ? a : v;
    r = b > r ? b : r;
  }
  const bool neg = __any_sync(0xffffffffu, negative);
  if ((threadIdx.x & 31) != 0) return;
  unsigned long long* F = S.fold;
  if (v) atomicMax(F + kFoldVel2, v);
  if (r) atomicMax(F + kFoldRate2, r);
  if (neg) atomicMax(F + kFoldNeg, 1ull);
  __threadfence();
  if (atomicAdd(F + kFoldDone, 1ull) != n_warps - 1) return;
  __threadfence();
  const double v2 = from_bits(atomicExch(F + kFoldVel2, 0ull)), r2 = from_bits(atomicExch(F + kFoldRate2, 0ull));
  const DtBounds b = dt_bounds(v2, r2, atomicExch(F + kFoldNeg, 0ull) != 0, P);
  atomicExch(F + kFoldDone, 0ull);
  S.scal[kScMaxVel] = b.max_vel;
  S.scal[kScExtraDt] = b.extra;
  S.scal[kScBound] = b.dt;
  S.scal[kScNegExtra] = b.negative ? 1.0 : 0.0;
}

__device__ __forceinline__ double step_dt(const double* scal, double dt0) { return clipped_dt(dt0, scal[kScBound]); }
// One thread of the step: its dt and time, and the stop bit of a negative
// extra dt, which the reference latches when the step begins.
__device__ __forceinline__ void publish_dt(const DevState& S, double dt) {
  S.scal[kScDt] = dt;
  if (S.dt_log) *S.dt_log = dt;
  S.scal[kScTime] = S.scal[kScTime] + dt;
  if (S.scal[kScNegExtra] != 0.0) atomicOr(S.err, 8u);  // SPLASH_STOP_NEG_EXTRA_DT
}
#endif

}  // namespace f64
}  // namespace splash
