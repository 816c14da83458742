// Host build of the FP64 path's limiter and Riemann fluxes, for CPU checks
// of the limiter's integer-comparison path against its general one and of
// the fluxes against the reference's known answers.
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

void flux(const double* uL, const double* uR, const double* ec, const double* en, double gam, int solver, double* F) {
  const D3 c = d3(ec[0], ec[1], ec[2]), n = d3(en[0], en[1], en[2]);
  const SlotGeom g{c, 1.0, n, cross3(n, c)};
  flux_star(uL, uR, g, gam, solver, F);
}

}  // extern "C"
