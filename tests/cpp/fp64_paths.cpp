// Host build of the FP64 path's limiter and Riemann fluxes, for CPU checks
// of the limiter's integer-comparison path against its general one and of
// the fluxes against the reference's known answers.
#include "limiter_pair.cuh"
#include "physics_fp64.cuh"

using namespace splash;
using namespace splash::f64;

extern "C" {

// both limiter paths on n cases: r, superbee scale, Courant factor
void limiter_both(int n, const double* r, const double* sb, const double* nu, double eta_p, double* general,
                  double* positive) {
  for (int i = 0; i < n; ++i) {
    const double ts = (1 + nu[i]) / 3;
    const LimiterLine<double> line{eta_p, sb[i], ts, 1 - ts};
    general[i] = limiter_field(r[i], line);
    positive[i] = limiter_field_pos(r[i], line);
  }
}

// the limiter in pairs of floats and in FP64 on n cases of dp, num, nu; served: 1 where pairs serve
void limiter_pairs(int n, const double* dp, const double* num, const double* nu, double eta_p, double sbs, double* pairs,
                   double* full, int* served) {
  for (int i = 0; i < n; ++i) {
    pairs[i] = 0.0;
    served[i] = limiter_pair(dp[i], num[i], dp[i] - num[i], pair_line(eta_p, sbs, nu[i]), pairs[i]);
    const double ts = (1 + nu[i]) / 3;
    full[i] = limiter_field(num[i] / dp[i], LimiterLine<double>{eta_p, sbs / nu[i], ts, 1 - ts});
  }
}

void flux(const double* uL, const double* uR, const double* ec, const double* en, double gam, int solver, double* F) {
  const D3 c = d3(ec[0], ec[1], ec[2]), n = d3(en[0], en[1], en[2]);
  const SlotGeom g{c, 1.0, n, cross3(n, c)};
  flux_star(uL, uR, g, gam, solver, F);
}

}  // extern "C"
