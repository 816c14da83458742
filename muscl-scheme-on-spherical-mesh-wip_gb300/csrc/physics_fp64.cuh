// FP64 device physics of the MUSCL step: pressures, edge velocities, the
// three Riemann solvers, the blended limiter, the accretion source and the
// dt candidates.
//
// Each function evaluates one reference function (cited) from the formulas
// it stands for, in a form that takes few FP64 instructions (fp64_math.cuh
// says why they are what counts): one reciprocal per state shared by its
// quotients, squared speeds instead of roots that are squared again, fused
// multiply-adds, only the side of the Riemann fan that the flux needs.  The
// functions are templates over the scalar type: `double` for the time step
// (the translation units that use them are compiled with -fmad=false, so
// nothing is fused but what is written so), and Dual<N> (dual.cuh) for the
// tangent-linear and adjoint kernels, whose values are computed by the same
// operations and so follow the same branches.
#pragma once

#include <cmath>
#include <type_traits>

#include "dual.cuh"
#include "fp64_math.cuh"
#include "layout.hpp"

namespace splash {
namespace f64 {

template <class T>
struct V3 {
  T x, y, z;
};
using D3 = V3<double>;

template <class T>
SPLASH_HD V3<T> v3(const T& x, const T& y, const T& z) {
  return V3<T>{x, y, z};
}
SPLASH_HD D3 d3(double x, double y, double z) { return D3{x, y, z}; }
template <class A, class B>
SPLASH_HD auto sub(const V3<A>& a, const V3<B>& b) -> V3<wider_t<A, B>> {
  return V3<wider_t<A, B>>{a.x - b.x, a.y - b.y, a.z - b.z};
}
template <class T, class S>
SPLASH_HD auto scal(const V3<T>& a, const S& s) -> V3<wider_t<T, S>> {
  return V3<wider_t<T, S>>{a.x * s, a.y * s, a.z * s};
}
template <class A, class B>
SPLASH_HD auto cross3(const V3<A>& a, const V3<B>& b) -> V3<wider_t<A, B>> {
  return V3<wider_t<A, B>>{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <class A, class B>
SPLASH_HD auto dot3(const V3<A>& a, const V3<B>& b) -> wider_t<A, B> {
  return a.x * b.x + a.y * b.y + a.z * b.z;
}
// the same with fused multiply-adds
template <class A, class B>
SPLASH_HD auto fcross(const V3<A>& a, const V3<B>& b) -> V3<wider_t<A, B>> {
  return V3<wider_t<A, B>>{fm(a.y, b.z, -(a.z * b.y)), fm(a.z, b.x, -(a.x * b.z)), fm(a.x, b.y, -(a.y * b.x))};
}
template <class A, class B>
SPLASH_HD auto fdot(const V3<A>& a, const V3<B>& b) -> wider_t<A, B> {
  return fm(a.z, b.z, fm(a.y, b.y, a.x * b.x));
}

// MUSCL_base.hpp:517-539 (u[4] = energy, r = unit face centre): with
// v = r x l / (-Sigma), Pi = max(1e-16, (E - |r x l|^2 / (2 Sigma)) (gam - 1))
template <class T>
SPLASH_HD T pressure_fc(const T* u, const D3& r, double gam) {
  const V3<T> c = fcross(r, v3(u[1], u[2], u[3]));
  return smax(T(1e-16), fm(-0.5 * fdot(c, c), recip(u[0]), u[4]) * (gam - 1));
}

// The constants of the gas that the fluxes use.
struct Gas {
  double gam, inv_gm1, shock_k;  // gam, 1 / (gam - 1), (gam + 1) / (2 gam)
};
SPLASH_HD Gas gas_of(const PhysParams& P) { return Gas{P.gam, P.inv_gm1, P.shock_k}; }

// Geometry of one edge as the flux sees it: unit edge centre, normal,
// cross(normal, centre).
struct EdgeGeom {
  D3 ec, en, nxr;
};

// One side of a Riemann problem from its limited edge state
// u = (Sigma, l, Pi): velocity ec x l / (-Sigma) (adiabatic.hpp:375-376),
// its normal component and square, the floored pressure (:582-592), the
// energy (MUSCL_base.hpp:541-562) and the sound speed.
template <class T>
struct EdgeSide {
  V3<T> vel;
  T vn, v2, p, e;
  T gi;     // gam / Sigma
  T a2, a;  // gam Pi / Sigma, its root
  T q;      // the wave speed relative to vn (char_vel), set by wave_speeds
};
template <class T>
SPLASH_HD EdgeSide<T> edge_side(const T* u, const EdgeGeom& g, const Gas& gas) {
  EdgeSide<T> S;
  const T ir = recip(u[0]);
  S.vel = scal(fcross(g.ec, v3(u[1], u[2], u[3])), -ir);
  S.vn = fdot(g.en, S.vel);
  S.v2 = fdot(S.vel, S.vel);
  S.p = smax(T(1e-16), u[4]);
  S.e = fm(0.5 * u[0], S.v2, gas.inv_gm1 * u[4]);
  S.gi = gas.gam * ir;
  S.a2 = S.gi * S.p;
  S.a = root(S.a2);
  return S;
}

// char_vel (physics/adiabatic.hpp:594-683): the distance of the outer wave
// from vn on each side, a sqrt(1 + k (p* / p - 1)) = sqrt(gam / Sigma
// (p + k (p* - p))) behind a shock and a otherwise (also where that is not
// finite).
template <class T>
SPLASH_HD T wave_speed(const EdgeSide<T>& S, const T& p_star, const Gas& gas) {
  if (!less(S.p, p_star)) return S.a;
  const T q = root(S.gi * fm(gas.shock_k, p_star - S.p, S.p));
  return odd_bits(val(q)) ? S.a : q;
}
template <class T>
SPLASH_HD T star_pressure(const T* uL, const T* uR, const EdgeSide<T>& L, const EdgeSide<T>& R) {
  const T pvrs = fm(-0.125 * ((R.vn - L.vn) * (uL[0] + uR[0])), L.a + R.a, 0.5 * (L.p + R.p));
  return smax(T(0.), pvrs);
}

// physics/adiabatic.hpp:352-392
template <class T>
SPLASH_HD void phys_flux(const T* u, const EdgeSide<T>& S, const EdgeGeom& g, T* F) {
  F[0] = u[0] * S.vn;
  F[1] = fm(u[1], S.vn, -(g.nxr.x * S.p));
  F[2] = fm(u[2], S.vn, -(g.nxr.y * S.p));
  F[3] = fm(u[3], S.vn, -(g.nxr.z * S.p));
  F[4] = (S.e + S.p) * S.vn;
}

// The HLLC+ factor f*(M) sqrt(4 + (1 - M^2)^2) M / (1 + M^2) of
// HLLCplus.hpp from M^2; M receives M.
template <class T>
SPLASH_HD T hllcp_fstar(const T& mm, T& M) {
  M = root(mm);
  const T om = 1.0 - mm;
  return M * root(fm(om, om, T(4.))) * recip(1.0 + mm);
}

// Riemann fluxes of the states uL, uR = (Sigma, l, Pi): HLLE_p.hpp:19-58
// (solver 1), HLLC.hpp:138-242 (solver 2), HLLCplus.hpp:17-177 (solver 3).
// Returns stop bits (STOP_NAN_WAVESPEED, STOP_WAVE_ORDER as in
// splash_gb300.h).
//
// The star-region flux F_K* = (S* (S_K u_K - F_K) + S_K P D) / (S_K - S*)
// (HLLC.hpp:218-239) is evaluated with F_K inserted: with
// s = S* / (S_K - S*), alpha = s (S_K - V_K) and beta = (S* p_K - S_K P) /
// (S_K - S*) = s (p_K - P) - P it is alpha Sigma, alpha l + beta (n x R) and
// alpha E + s (S_K P - p_K V_K), 2 instructions per momentum component, of
// the one side that S* selects.
//
// L and R are the edge_side of the states (their q is not read).
template <class T>
SPLASH_HD unsigned riemann_flux(const T* uL, const T* uR, EdgeSide<T> L, EdgeSide<T> R, const EdgeGeom& g,
                                const Gas& gas, int solver, T* F) {
  unsigned bits = 0;
  const T p_star = star_pressure(uL, uR, L, R);
  L.q = wave_speed(L, p_star, gas);
  R.q = wave_speed(R, p_star, gas);
  const T S_L = L.vn - L.q, S_R = R.vn + R.q;
  if (nan_bits(val(S_L)) || nan_bits(val(S_R))) bits |= 2u;
  if (solver == 1) {
    if (not_below_zero(S_L)) {
      phys_flux(uL, L, g, F);
    } else if (below_zero(S_L) && below_zero(-S_R)) {
      T FL[kDim], FR[kDim];
      phys_flux(uL, L, g, FL);
      phys_flux(uR, R, g, FR);
      // (S_R F_L - S_L F_R + S_R S_L (u_R - u_L)) / (S_R - S_L) around F_R,
      // so that the quotient's rounding only meets differences
      const T wl = S_R * recip(S_R - S_L);
      const T t = wl * S_L;
#pragma unroll
      for (int i = 0; i < kDim; ++i) {
        const T du = (i < 4) ? uR[i] - uL[i] : R.e - L.e;
        F[i] = fm(wl, FL[i] - FR[i], fm(t, du, FR[i]));
      }
    } else {
      // S_R <= 0, or NaN wave speeds (reference prints and stops)
      if (!not_below_zero(-S_R)) bits |= 4u;
      phys_flux(uR, R, g, F);
    }
    return bits;
  }
  // phi = Sigma (S - V) of each side
  const T mL = -(uL[0] * L.q), mR = uR[0] * R.q;
  const T iden = recip(mL - mR);
  T S_star = fm(L.vn, mL, fm(-R.vn, mR, R.p - L.p)) * iden;
  if (odd_bits(val(S_star))) S_star = 0.5 * (L.vn + R.vn);
  // branch choice of HLLC.hpp:218-239 / HLLCplus.hpp:153-174
  int side;  // 0: F_L, 1: F_L*, 2: F_R*, 3: F_R
  if (not_below_zero(S_L)) {
    side = 0;
  } else if (below_zero(S_L) && not_below_zero(S_star)) {
    side = 1;
  } else if (below_zero(S_star) && not_below_zero(S_R)) {
    side = 2;
  } else {
    if (!below_zero(S_R)) bits |= 4u;
    side = 3;
  }
  if (side == 0) {
    phys_flux(uL, L, g, F);
    return bits;
  }
  if (side == 3) {
    phys_flux(uR, R, g, F);
    return bits;
  }
  const bool left = side == 1;
  const T P_LR = 0.5 * fm(mR, S_star - R.vn, fm(mL, S_star - L.vn, L.p + R.p));
  const T Sk = left ? S_L : S_R;
  const T inv = recip(Sk - S_star);
  {
    const T pk = left ? L.p : R.p;
    const T si = S_star * inv;
    const T al = si * (left ? -L.q : R.q);
    const T be = fm(si, pk - P_LR, -P_LR);
    F[0] = al * (left ? uL[0] : uR[0]);
    F[1] = fm(al, left ? uL[1] : uR[1], be * g.nxr.x);
    F[2] = fm(al, left ? uL[2] : uR[2], be * g.nxr.y);
    F[3] = fm(al, left ? uL[3] : uR[3], be * g.nxr.z);
    F[4] = fm(al, left ? L.e : R.e, si * fm(Sk, P_LR, -(pk * (left ? L.vn : R.vn))));
  }
  if (solver == 3) {
    // M^2 = min(1, max(|v|^2 / a^2)); the larger quotient by cross products
    const bool rfast = less(L.v2 * R.a2, R.v2 * L.a2);
    T mm = divide(rfast ? R.v2 : L.v2, rfast ? R.a2 : L.a2);
    if (!less(mm, T(1.))) mm = T(1.);
    T M;
    T f1 = hllcp_fstar(mm, M) - 1.0;
    // sonic points (HLLCplus.hpp:96-107) need |v| >= a on some side
    if (!less_pos(val(mm), 0.999)) {
      const T lm = L.vn - L.a, lp = L.vn + L.a, rm = R.vn - R.a, rp = R.vn + R.a;
      if ((lm > 0 && rm < 0) || (lp > 0 && rp < 0) || (rm > 0 && lm < 0) || (rp > 0 && lp < 0)) f1 = T(0.);
    }
    const T gsw = pressure_switch(M, L.p, R.p);
    const T dV = R.vn - L.vn;
    const T cs = Sk * inv * gsw;
    // ec x (f1 dV n + cs (dv - dV n)), with ec x n = -(n x ec)
    const T k1 = (cs - f1) * dV;
    const V3<T> ed = fcross(g.ec, sub(R.vel, L.vel));
    const T w = -(mL * mR) * iden;
    F[1] = fm(w, fm(cs, ed.x, k1 * g.nxr.x), F[1]);
    F[2] = fm(w, fm(cs, ed.y, k1 * g.nxr.y), F[2]);
    F[3] = fm(w, fm(cs, ed.z, k1 * g.nxr.z), F[3]);
    F[4] = fm(w, f1 * dV * S_star, F[4]);
  }
  return bits;
}

template <class T>
SPLASH_HD unsigned riemann_flux(const T* uL, const T* uR, const EdgeGeom& g, const Gas& gas, int solver, T* F) {
  return riemann_flux(uL, uR, edge_side(uL, g, gas), edge_side(uR, g, gas), g, gas, solver, F);
}

// Geometry of one slot with the edge centre as evaluated (not exactly unit).
struct SlotGeom {
  D3 ec;       // unit edge centre
  double ecn;  // |ec|
  D3 en;       // edge normal
  D3 nxr;      // cross(en, ec/|ec|)
};
SPLASH_HD EdgeGeom edge_geom(const SlotGeom& g) {
  return EdgeGeom{d3(g.ec.x / g.ecn, g.ec.y / g.ecn, g.ec.z / g.ecn), g.en, g.nxr};
}
SPLASH_HD Gas gas_of(double gam) { return Gas{gam, 1 / (gam - 1), (gam + 1) / (2 * gam)}; }
// Pi of a conserved state (u[4] = energy) at the edge
template <class T>
SPLASH_HD T edge_pressure(const T* u, const EdgeGeom& g, double gam) {
  const V3<T> c = fcross(g.ec, v3(u[1], u[2], u[3]));
  return fm(-0.5 * fdot(c, c), recip(u[0]), u[4]) * (gam - 1);
}
// riemann_flux of two conserved states (u[4] = energy)
template <class T>
SPLASH_HD unsigned flux_star(const T* uL, const T* uR, const SlotGeom& sg, double gam, int solver, T* F) {
  const EdgeGeom g = edge_geom(sg);
  const T L[kDim] = {uL[0], uL[1], uL[2], uL[3], edge_pressure(uL, g, gam)};
  const T R[kDim] = {uR[0], uR[1], uR[2], uR[3], edge_pressure(uR, g, gam)};
  return riemann_flux(L, R, g, gas_of(gam), solver, F);
}

// What one slot's limiter shares over the fields: eta_plus = H+/BM, the
// superbee scale eta_minus / (2 N nu) and the third-order line
// 1 + (1 + nu)/3 (r - 1) = t1 + ts r (physics/adiabatic.hpp:741-828).
template <class T>
struct LimiterLine {
  double eta_p;
  T sb, ts, t1;
};

// physics/adiabatic.hpp:685-828 for one field: blend of the third-order
// limiter and the irregular-grid superbee, NaN ratio -> 0.  Where the two
// limiters agree the blend is their value whatever the switch; the switch is
// evaluated only where they differ.
template <class T>
SPLASH_HD T limiter_field(const T& r, const LimiterLine<T>& l) {
  if (is_nan(r)) return T(0.);
  const T sb = smax(T(0.), smax(smin(T(1.), r * l.sb), smin(r, T(l.eta_p))));
  const T to = smax(T(0.), smin(sb, fm(l.ts, r, l.t1)));
  if (val(to) == val(sb)) return sb;
  if (!(val(r) > 0.0)) return to;
  return fm(switch_pos(val(r)), sb - to, to);
}
// The same for a positive, finite superbee scale (nu > 0: no supersonic
// inflow) on integer comparisons alone: then every operand of the min and max
// is non-negative where r is, and the limiter is 0 where it is not.
SPLASH_HD double limiter_field_pos(double r, const LimiterLine<double>& l) {
  const int64_t rb = (int64_t)bits_of(r);
  if (rb <= 0 || rb > 0x7ff0000000000000ll) return 0.0;
  const double rs = r * l.sb;
  const double A = less_pos(rs, 1.0) ? rs : 1.0;
  const double B = less_pos(l.eta_p, r) ? l.eta_p : r;
  const double sb = less_pos(A, B) ? B : A;
  const double t = fma(l.ts, r, l.t1);
  if ((int64_t)bits_of(t) < 0) return fma(switch_pos(r), sb, 0.0);
  if (!less_pos(t, sb)) return sb;
  return fma(switch_pos(r), sb - t, t);
}

// The candidates of one face for the next dt (find_v_max,
// MUSCL_base.hpp:311-343; extra_dt_constr, physics/adiabatic.hpp:543-580) in
// the form in which they are folded (FoldSlot): the larger of |v|^2 and the squared sound speed, and
// rate2 = (g_eff Sigma |v - v0| / Pi)^2, the squared reciprocal of the extra
// dt 0.01 Pi / (alpha fric_k g_eff Sigma |v - v0|) but for the constant factor
// (no root and no quotient but 1 / Sigma and 1 / Pi per face).  `negative`
// reports a negative extra dt, by the signs of g_eff Sigma / Pi and of alpha
// (a zero counts by its sign: it makes the extra dt infinite); NaN candidates
// are 0, like the reference's comparisons skip them.  w holds (Sigma, l, Pi).
SPLASH_HD void dt_fold(const double* w, const D3& r, const PhysParams& P, double& vel2, double& rate2,
                       bool& negative) {
  const double ir = recip(w[0]);
  const D3 vel = scal(fcross(r, d3(w[1], w[2], w[3])), -ir);
  const double v2 = fdot(vel, vel);
  const double a2 = P.gam * (w[4] * ir);
  const D3 rel = d3(fma(P.omega_ns, r.y, vel.x), fma(-P.omega_ns, r.x, vel.y), vel.z);
  const double n2 = fdot(rel, rel);
  const double GM = 0.217909;
  const double t = (GM - v2) * w[0] * recip(w[4]);
  vel2 = 0.0;
  if (!nan_bits(v2)) vel2 = v2;
  if (not_below_zero(a2) && less_pos(vel2, a2)) vel2 = a2;
  rate2 = t * t * n2;
  negative = (high_word(t) ^ high_word(P.alpha)) >> 31 && !odd_bits(t) && !odd_bits(n2);
  if (nan_bits(rate2)) rate2 = 0.0;
}

// The parameters of the source term that the derivative kernels
// differentiate: the face's accretion profile value acc0 (res[0] of
// physics/adiabatic.hpp:415-421), the accretion angular velocity, the
// accretion rate and the initial total mass (both enter the depletion term
// without friction).
template <class Q>
struct SrcParams {
  Q acc0;
  V3<Q> omega_acc;
  Q acc_rate;
  Q total_mass;
};

// physics/adiabatic.hpp:396-541 ; w[4] is the pressure.
template <class T, class Q>
SPLASH_HD void source_term(const T* w, const D3& fcn, const SrcParams<Q>& sp, const PhysParams& P, T* res) {
  const Q& acc0 = sp.acc0;
  const V3<Q>& omega_acc = sp.omega_acc;
#pragma unroll
  for (int i = 0; i < kDim; ++i) res[i] = T(0.);
  if (!P.accretion_on) return;
  const T ir = recip(w[0]);
  const V3<T> vel = scal(fcross(fcn, v3(w[1], w[2], w[3])), -ir);
  const T v2 = fdot(vel, vel);
  res[0] = T(acc0);
  const V3<Q> omxr = fcross(omega_acc, fcn);
  const V3<Q> rxo = fcross(fcn, omxr);
  res[1] = res[0] * rxo.x;
  res[2] = res[0] * rxo.y;
  res[3] = res[0] * rxo.z;
  const V3<T> d = v3(T(omxr.x - vel.x), T(omxr.y - vel.y), T(omxr.z - vel.z));
  res[4] = res[0] * fm(0.5, fdot(d, d), T(P.e_acc));
  if (!P.friction_on) {
    const V3<T> rxv = fcross(fcn, vel);
    const double fall_eff = 1;
    const T dmdt = divide(-(fall_eff * sp.acc_rate * (4 * M_PI)), sp.total_mass) * w[0];
    res[0] += dmdt;
    res[1] = fm(dmdt, rxv.x, res[1]);
    res[2] = fm(dmdt, rxv.y, res[2]);
    res[3] = fm(dmdt, rxv.z, res[3]);
    res[4] = fm(dmdt, fm(P.gam_gm1 * w[4], ir, 0.5 * v2), res[4]);
  }
  const double GM = 0.217909;
  const T g_eff = GM - v2;
  const double c_sigma = 4.85e36;
  const double k_m = 1.6e-13;
  const double kappa = 3.4e6;
  const T ip = recip(w[4]);
  const T C = (12. / 5 * k_m) * (w[0] * ip) * root(root((3. / 4 * c_sigma) * (g_eff * w[0])));
  const double beta_switch = 0.736194670678821;
  const double C_switch = -1 - 1 / (beta_switch - 1);
  T beta;
  if (C <= C_switch) {
    beta = 1.0 - recip(1.0 + C);
  } else {
    const T x = 2.0 * recip(C), x2 = x * x;
    beta = 1.0 - x2 * x2;
  }
  const double beta_ceil = 1 - 1e-8, beta_floor = 1e-8;
  if (beta < beta_floor || is_nan(beta)) beta = T(beta_floor);
  if (beta > beta_ceil) beta = T(beta_ceil);
  res[4] -= g_eff * (1 / kappa) * (1.0 - beta);
  if (P.friction_on) {
    const T rho = P.fric_k * g_eff * w[0] * w[0] * ip;  // fric_k = gam3d / (2 gam3d - 1)
    const D3 vel0 = d3(-P.omega_ns * fcn.y, P.omega_ns * fcn.x, 0.0);  // (0, 0, omega_ns) x fcn
    const V3<T> rel = sub(vel, vel0);
    const T k = P.alpha * rho * root(fdot(rel, rel));
    const V3<T> wr = scal(rel, -k);
    const V3<T> l_fr = fcross(fcn, wr);
    const T kr = k * ir;
    res[0] -= k;
    res[1] = fm(-kr, w[1], res[1] + l_fr.x);
    res[2] = fm(-kr, w[2], res[2] + l_fr.y);
    res[3] = fm(-kr, w[3], res[3] + l_fr.z);
    res[4] = fm(-k, fm(P.gam_gm1 * w[4], ir, 0.5 * v2), res[4] + fdot(wr, vel0));
  }
}

}  // namespace f64
}  // namespace splash
