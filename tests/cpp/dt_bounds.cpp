// Host build of the FP64 path's dt clip: the faces' candidates folded as the
// kernels fold them, and the bounds that are made of the folds.
#include "step_fold_fp64.cuh"
#include "physics_fp64.cuh"

using namespace splash;

// w: n states (Sigma, l, Pi), r: n unit face centres; out: max_vel, extra dt, the bound of dt, 1 where the step stops
extern "C" void dt_bounds_of(int n, const double* w, const double* r, double gam, double omega_ns, double alpha, double h0,
                             double* out) {
  PhysParams P{};
  P.gam = gam;
  P.omega_ns = omega_ns;
  P.alpha = alpha;
  P.h0 = h0;
  derive_params(P);
  double vel2 = 0.0, rate2 = 0.0;
  bool negative = false;
  for (int i = 0; i < n; ++i) {
    double v, q;
    bool neg;
    f64::dt_fold(w + 5 * i, f64::d3(r[3 * i], r[3 * i + 1], r[3 * i + 2]), P, v, q, neg);
    vel2 = v > vel2 ? v : vel2;
    rate2 = q > rate2 ? q : rate2;
    negative = negative || neg;
  }
  const f64::DtBounds b = f64::dt_bounds(vel2, rate2, negative, P);
  out[0] = b.max_vel;
  out[1] = b.extra;
  out[2] = b.dt;
  out[3] = b.negative ? 1.0 : 0.0;
}
