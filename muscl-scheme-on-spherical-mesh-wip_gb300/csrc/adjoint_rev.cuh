// Reverse (adjoint) forms of the FP64 per-slot and per-face physics.
//
// Each reverse function recomputes the primal with exactly the operations
// of physics_fp64.cuh (so it takes the same branches as the forward step:
// limiter cases, wave-speed sides, HLLC+ switches, floors) and then
// propagates the adjoint of its outputs back to its inputs.  Conventions:
// `xb` is the adjoint (bar) of x; reverse functions ADD into the bars of
// their inputs.  At a kink the derivative of the branch taken is used,
// matching the forward-mode duals of dual.cuh.
//
//   riemann_flux_rev  hand-written reverse of the three Riemann solvers
//                     (HLLE_p.hpp:19-58, HLLC.hpp:138-242,
//                     HLLCplus.hpp:17-177, char_vel adiabatic.hpp:594-683)
//   recon_side_tape   find_U_edges (MUSCL_base.hpp:361-434) of one side with
//                     the local limiter Jacobian (adiabatic.hpp:685-828) taped
//   recon_side_rev    reverse of the reconstruction from that tape
//   source_rev        reverse of the source term (adiabatic.hpp:396-541)
//                     in its 5 state and 5 parameter inputs
//   prim_rev          reverse of (Sigma, l, E) -> (Sigma, l, Pi)
#pragma once

#include "dual.cuh"
#include "physics_fp64.cuh"
#include "step_body_fp64.cuh"

namespace splash {
namespace f64 {
namespace rev {

// ---------------------------------------------------------------------
// Adjoints of the quantities of one side of a Riemann problem (EdgeSide).
struct SideBar {
  double u0, u4, vn, v2, p, e, gi, a2, a, q;
  D3 l, vel;
};
SPLASH_HD void zero(SideBar& b) {
  b.u0 = b.u4 = b.vn = b.v2 = b.p = b.e = b.gi = b.a2 = b.a = b.q = 0.0;
  b.l = b.vel = d3(0, 0, 0);
}
// a SideBar as values at p[0], p[stride], ... (q is folded into the others
// before it is handed on)
constexpr int kSideBarValues = 15;
SPLASH_HD void put_bar(double* p, int stride, const SideBar& b) {
  const double v[kSideBarValues] = {b.u0, b.u4, b.vn, b.v2, b.p, b.e, b.gi, b.a2, b.a, b.l.x, b.l.y, b.l.z,
                                    b.vel.x, b.vel.y, b.vel.z};
  for (int i = 0; i < kSideBarValues; ++i) p[(size_t)i * stride] = v[i];
}
SPLASH_HD SideBar get_bar(const double* p, int stride) {
  double v[kSideBarValues];
  for (int i = 0; i < kSideBarValues; ++i) v[i] = p[(size_t)i * stride];
  SideBar b;
  b.u0 = v[0];
  b.u4 = v[1];
  b.vn = v[2];
  b.v2 = v[3];
  b.p = v[4];
  b.e = v[5];
  b.gi = v[6];
  b.a2 = v[7];
  b.a = v[8];
  b.q = 0.0;
  b.l = d3(v[9], v[10], v[11]);
  b.vel = d3(v[12], v[13], v[14]);
  return b;
}
SPLASH_HD void add_scaled(D3& a, const D3& b, double s) {
  a.x = fma(b.x, s, a.x);
  a.y = fma(b.y, s, a.y);
  a.z = fma(b.z, s, a.z);
}

// Reverse of phys_flux
SPLASH_HD void phys_flux_rev(const double* u, const EdgeSide<double>& S, const EdgeGeom& g, const double* Fb,
                             SideBar& B) {
  const D3 lb = d3(Fb[1], Fb[2], Fb[3]);
  B.u0 = fma(Fb[0], S.vn, B.u0);
  B.vn += fma(Fb[4], S.e + S.p, fma(Fb[0], u[0], fdot(lb, d3(u[1], u[2], u[3]))));
  add_scaled(B.l, lb, S.vn);
  B.p += fma(Fb[4], S.vn, -fdot(g.nxr, lb));
  B.e = fma(Fb[4], S.vn, B.e);
}

// Reverse of edge_side: the adjoint of (Sigma, l, Pi)
SPLASH_HD void edge_side_rev(const double* u, const EdgeSide<double>& S, const EdgeGeom& g, const Gas& gas,
                             SideBar& B, double* ub) {
  // a = sqrt(a2), a2 = gi p
  if (S.a > 0.0) B.a2 = fma(B.a * 0.5, recip(S.a), B.a2);
  B.gi = fma(B.a2, S.p, B.gi);
  B.p = fma(B.a2, S.gi, B.p);
  // e = Sigma v2 / 2 + Pi / (gam - 1), p = max(1e-16, Pi)
  B.u0 = fma(0.5 * S.v2, B.e, B.u0);
  B.v2 = fma(0.5 * u[0], B.e, B.v2);
  B.u4 = fma(gas.inv_gm1, B.e, B.u4);
  if (less(1e-16, u[4])) B.u4 += B.p;
  add_scaled(B.vel, S.vel, 2 * B.v2);
  add_scaled(B.vel, g.en, B.vn);
  // vel = -(ec x l) / Sigma, gi = gam / Sigma
  const double ir = recip(u[0]);
  const D3 cb = scal(B.vel, -ir);
  B.u0 -= ir * fma(B.gi, S.gi, fdot(B.vel, S.vel));
  const D3 lb = fcross(cb, g.ec);
  ub[0] += B.u0;
  ub[1] += B.l.x + lb.x;
  ub[2] += B.l.y + lb.y;
  ub[3] += B.l.z + lb.z;
  ub[4] += B.u4;
}

// Reverse of wave_speed; returns the adjoint of p_star
SPLASH_HD double wave_speed_rev(const EdgeSide<double>& S, double p_star, const Gas& gas, SideBar& B) {
  if (less(S.p, p_star)) {
    const double z = fma(gas.shock_k, p_star - S.p, S.p);
    const double q = root(S.gi * z);
    if (!odd_bits(q)) {
      const double qq = B.q * 0.5 * recip(q);
      B.gi = fma(qq, z, B.gi);
      const double zb = qq * S.gi;
      B.p = fma(zb, 1 - gas.shock_k, B.p);
      return zb * gas.shock_k;
    }
  }
  B.a += B.q;
  return 0.0;
}

// Adjoint of F = riemann_flux(uL, uR, L, R): the adjoints of the two sides'
// quantities (edge_side_rev turns them into those of the states).
SPLASH_HD void riemann_flux_rev(const double* uL, const double* uR, EdgeSide<double> L, EdgeSide<double> R,
                                const EdgeGeom& g, const Gas& gas, int solver, const double* Fb, SideBar& BL,
                                SideBar& BR) {
  const double pvrs = fma(-0.125 * ((R.vn - L.vn) * (uL[0] + uR[0])), L.a + R.a, 0.5 * (L.p + R.p));
  const double p_star = smax(0., pvrs);
  L.q = wave_speed(L, p_star, gas);
  R.q = wave_speed(R, p_star, gas);
  const double S_L = L.vn - L.q, S_R = R.vn + R.q;
  zero(BL);
  zero(BR);
  double SLb = 0.0, SRb = 0.0;

  if (solver == 1) {
    if (not_below_zero(S_L)) {
      phys_flux_rev(uL, L, g, Fb, BL);
    } else if (below_zero(S_L) && below_zero(-S_R)) {
      double FL[kDim], FR[kDim], FLb[kDim], FRb[kDim];
      phys_flux(uL, L, g, FL);
      phys_flux(uR, R, g, FR);
      const double inv = recip(S_R - S_L);
      const double wl = S_R * inv;
      const double t = wl * S_L;
      double wb = 0.0, tb = 0.0, dub[kDim];
#pragma unroll
      for (int i = 0; i < kDim; ++i) {
        const double du = (i < 4) ? uR[i] - uL[i] : R.e - L.e;
        wb = fma(Fb[i], FL[i] - FR[i], wb);
        tb = fma(Fb[i], du, tb);
        FLb[i] = wl * Fb[i];
        FRb[i] = Fb[i] - FLb[i];
        dub[i] = t * Fb[i];
      }
      // wl = S_R inv, t = wl S_L, inv = 1 / (S_R - S_L)
      wb = fma(tb, S_L, wb);
      SLb = fma(tb, wl, SLb);
      SRb = fma(wb, inv, SRb);
      const double db = -(wb * S_R) * inv * inv;
      SRb += db;
      SLb -= db;
      BR.u0 += dub[0];
      BL.u0 -= dub[0];
      add_scaled(BR.l, d3(dub[1], dub[2], dub[3]), 1.0);
      add_scaled(BL.l, d3(dub[1], dub[2], dub[3]), -1.0);
      BR.e += dub[4];
      BL.e -= dub[4];
      phys_flux_rev(uL, L, g, FLb, BL);
      phys_flux_rev(uR, R, g, FRb, BR);
    } else {
      phys_flux_rev(uR, R, g, Fb, BR);
    }
  } else {
    const double mL = -(uL[0] * L.q), mR = uR[0] * R.q;
    const double iden = recip(mL - mR);
    const double num = fma(L.vn, mL, fma(-R.vn, mR, R.p - L.p));
    double S_star = num * iden;
    const bool mean = odd_bits(S_star);
    if (mean) S_star = 0.5 * (L.vn + R.vn);
    int side;
    if (not_below_zero(S_L))
      side = 0;
    else if (below_zero(S_L) && not_below_zero(S_star))
      side = 1;
    else if (below_zero(S_star) && not_below_zero(S_R))
      side = 2;
    else
      side = 3;
    if (side == 0) {
      phys_flux_rev(uL, L, g, Fb, BL);
    } else if (side == 3) {
      phys_flux_rev(uR, R, g, Fb, BR);
    } else {
      const bool left = (side == 1);
      const double P_LR = 0.5 * fma(mR, S_star - R.vn, fma(mL, S_star - L.vn, L.p + R.p));
      const double Sk = left ? S_L : S_R;
      const double inv = recip(Sk - S_star);
      const double* uk = left ? uL : uR;
      const EdgeSide<double>& K = left ? L : R;
      SideBar& BK = left ? BL : BR;
      const double si = S_star * inv;
      const double qk = left ? -L.q : R.q;
      const double al = si * qk;
      double Skb = 0.0, Ssb = 0.0, invb = 0.0, mLb = 0.0, mRb = 0.0, idenb = 0.0;
      const D3 lb = d3(Fb[1], Fb[2], Fb[3]);
      if (solver == 3) {
        const bool rfast = less(L.v2 * R.a2, R.v2 * L.a2);
        double mm = divide(rfast ? R.v2 : L.v2, rfast ? R.a2 : L.a2);
        const bool capped = !less(mm, 1.);
        if (capped) mm = 1.;
        Dual<1> Md;
        const Dual<1> fd = hllcp_fstar(Dual<1>::seed(mm, 0), Md);
        double f1 = fd.v - 1.0, df1 = fd.d[0];
        if (!less_pos(mm, 0.999)) {
          const double lm = L.vn - L.a, lp = L.vn + L.a, rm = R.vn - R.a, rp = R.vn + R.a;
          if ((lm > 0 && rm < 0) || (lp > 0 && rp < 0) || (rm > 0 && lm < 0) || (rp > 0 && lp < 0)) f1 = df1 = 0.;
        }
        const Dual<3> gd = pressure_switch(Dual<3>::seed(Md.v, 0), Dual<3>::seed(L.p, 1), Dual<3>::seed(R.p, 2));
        const double dV = R.vn - L.vn;
        const double cs = Sk * inv * gd.v;
        const double k1 = (cs - f1) * dV;
        const D3 ed = fcross(g.ec, sub(R.vel, L.vel));
        const double w = -(mL * mR) * iden;
        // F_l += w (k1 nxr + cs ed), F_E += w f1 dV S*
        const double lbn = fdot(lb, g.nxr), lbe = fdot(lb, ed);
        const double X = f1 * dV * S_star;
        const double wb = fma(Fb[4], X, fma(k1, lbn, cs * lbe));
        const double Xb = w * Fb[4];
        const double k1b = w * lbn;
        const double csb = fma(k1b, dV, w * lbe);
        const D3 dvb = fcross(scal(lb, w * cs), g.ec);
        add_scaled(BR.vel, dvb, 1.0);
        add_scaled(BL.vel, dvb, -1.0);
        const double f1b = fma(Xb * dV, S_star, -(k1b * dV));
        const double dVb = fma(Xb * f1, S_star, k1b * (cs - f1));
        Ssb = fma(Xb * f1, dV, Ssb);
        BR.vn += dVb;
        BL.vn -= dVb;
        Skb = fma(csb * inv, gd.v, Skb);
        invb = fma(csb * Sk, gd.v, invb);
        const double gb = csb * Sk * inv;
        BL.p = fma(gb, gd.d[1], BL.p);
        BR.p = fma(gb, gd.d[2], BR.p);
        if (!capped) {
          const double mmb = fma(f1b, df1, gb * gd.d[0] * Md.d[0]);
          const double ia = recip(rfast ? R.a2 : L.a2);
          SideBar& BF = rfast ? BR : BL;
          BF.v2 = fma(mmb, ia, BF.v2);
          BF.a2 = fma(-mmb * mm, ia, BF.a2);
        }
        mLb = fma(-wb * mR, iden, mLb);
        mRb = fma(-wb * mL, iden, mRb);
        idenb = fma(-wb * mL, mR, idenb);
      }
      // F_K* = (alpha Sigma, alpha l + beta nxr, alpha E + si (Sk P - p V))
      const double alb = fma(Fb[4], K.e, fma(Fb[0], uk[0], fdot(lb, d3(uk[1], uk[2], uk[3]))));
      BK.u0 = fma(Fb[0], al, BK.u0);
      add_scaled(BK.l, lb, al);
      BK.e = fma(Fb[4], al, BK.e);
      const double t = fma(Sk, P_LR, -(K.p * K.vn));
      const double beb = fdot(lb, g.nxr);
      const double sib = fma(beb, K.p - P_LR, fma(alb, qk, Fb[4] * t));
      const double tb = Fb[4] * si;
      const double qkb = alb * si;
      BK.p += fma(beb, si, -(tb * K.vn));
      BK.vn = fma(-tb, K.p, BK.vn);
      Skb = fma(tb, P_LR, Skb);
      const double Pb = 0.5 * (fma(tb, Sk, -beb) - beb * si);
      Ssb = fma(sib, inv, Ssb);
      invb = fma(sib, S_star, invb);
      // inv = 1 / (Sk - S*)
      const double db = -invb * inv * inv;
      Skb += db;
      Ssb -= db;
      if (left) {
        BL.q -= qkb;
        SLb += Skb;
      } else {
        BR.q += qkb;
        SRb += Skb;
      }
      // P_LR
      BL.p += Pb;
      BR.p += Pb;
      mLb = fma(Pb, S_star - L.vn, mLb);
      mRb = fma(Pb, S_star - R.vn, mRb);
      Ssb = fma(Pb, mL + mR, Ssb);
      BL.vn = fma(-Pb, mL, BL.vn);
      BR.vn = fma(-Pb, mR, BR.vn);
      // S* = num iden
      if (mean) {
        BL.vn = fma(0.5, Ssb, BL.vn);
        BR.vn = fma(0.5, Ssb, BR.vn);
      } else {
        const double numb = Ssb * iden;
        idenb = fma(Ssb, num, idenb);
        BR.p += numb;
        BL.p -= numb;
        BL.vn = fma(numb, mL, BL.vn);
        mLb = fma(numb, L.vn, mLb);
        BR.vn = fma(-numb, mR, BR.vn);
        mRb = fma(-numb, R.vn, mRb);
      }
      const double denb = -idenb * iden * iden;
      mLb += denb;
      mRb -= denb;
      BL.u0 = fma(-mLb, L.q, BL.u0);
      BL.q = fma(-mLb, uL[0], BL.q);
      BR.u0 = fma(mRb, R.q, BR.u0);
      BR.q = fma(mRb, uR[0], BR.q);
    }
  }
  // S_L = vn_L - q_L ; S_R = vn_R + q_R
  BL.vn += SLb;
  BL.q -= SLb;
  BR.vn += SRb;
  BR.q += SRb;
  const double psb = wave_speed_rev(L, p_star, gas, BL) + wave_speed_rev(R, p_star, gas, BR);
  const double ppb = less(0., pvrs) ? psb : 0.0;
  BL.p = fma(0.5, ppb, BL.p);
  BR.p = fma(0.5, ppb, BR.p);
  {
    const double t = -ppb * 0.125;
    const double dvn = R.vn - L.vn, rs = uL[0] + uR[0], as = L.a + R.a;
    const double dvnb = t * rs * as, rsb = t * dvn * as, asb = t * dvn * rs;
    BR.vn += dvnb;
    BL.vn -= dvnb;
    BL.u0 += rsb;
    BR.u0 += rsb;
    BL.a += asb;
    BR.a += asb;
  }
}

// Adjoint of flux_star (states with the energy in field 4)
SPLASH_HD void flux_star_rev(const double* uL, const double* uR, const SlotGeom& sg, double gam, int solver,
                             const double* Fb, double* uLb, double* uRb) {
  const EdgeGeom g = edge_geom(sg);
  Dual<5> pL, pR;
  const double* us[2] = {uL, uR};
  double st[2][kDim], bar[2][kDim] = {{0, 0, 0, 0, 0}, {0, 0, 0, 0, 0}};
  Dual<5>* ps[2] = {&pL, &pR};
  for (int i = 0; i < 2; ++i) {
    Dual<5> ud[kDim];
    for (int k = 0; k < kDim; ++k) ud[k] = Dual<5>::seed(us[i][k], k);
    *ps[i] = edge_pressure(ud, g, gam);
    for (int k = 0; k < 4; ++k) st[i][k] = us[i][k];
    st[i][4] = ps[i]->v;
  }
  const Gas gas = gas_of(gam);
  const EdgeSide<double> L = edge_side(st[0], g, gas), R = edge_side(st[1], g, gas);
  SideBar BL, BR;
  riemann_flux_rev(st[0], st[1], L, R, g, gas, solver, Fb, BL, BR);
  edge_side_rev(st[0], L, g, gas, BL, bar[0]);
  edge_side_rev(st[1], R, g, gas, BR, bar[1]);
  double* out[2] = {uLb, uRb};
  for (int i = 0; i < 2; ++i)
    for (int k = 0; k < kDim; ++k) out[i][k] += (k < 4 ? bar[i][k] : 0.0) + bar[i][4] * ps[i]->d[k];
}

// ---------------------------------------------------------------------
// Reconstruction with its reverse-sweep tape, and the reverse from the tape.
//
// Per side and field the limited edge state is up = w + hg dp phi(r, nu)
// with dp = U+ - w, dm = w - U-, r = hr dm / dp (hr = H+/H-, hg = BM/H+)
// and nu the side's Courant factor (MUSCL_base.hpp:361-434,
// adiabatic.hpp:685-828).  The recomputation evaluates phi with its two
// partial derivatives -- its value is the primal's, bit for bit -- and stores
//   d up / d dp = hg (phi - r phi_r),  d up / d dm = hg hr phi_r,
//   d up / d nu = hg dp phi_nu
// so that the reverse sweep needs no transcendental.  Where phi is flat in r
// (r = +-inf or NaN) d up / d dp = hg phi.
constexpr int kTapePlanes = 15;  // 3 per field

// field k; lj(3 k + i) receives its partials
template <class LjFn>
SPLASH_HD double limited_tape(const SideGeom& g, const SideLimiterPartials& limiter, int k, double w, double dp,
                              double dm, LjFn lj) {
  const double num = dm * g.hr, dpg = dp * g.hg;
  double r;
  const Phi phi = limiter(k, dp, num, dpg, r);
  lj(3 * k, g.hg * ((phi.r != 0.0) ? fma(-phi.r, r, phi.v) : phi.v));
  lj(3 * k + 1, g.hg * g.hr * phi.r);
  lj(3 * k + 2, dpg * phi.nu);
  return fm(dpg, phi.v, w);
}
// nb as in recon_side
template <class NbFn, class LjFn>
SPLASH_HD void recon_side_tape(const SideGeom& g, double gam, double dt, const double* w, NbFn nb, double* up,
                               LjFn lj) {
  double c;
  const double nu = side_courant(g, gam, dt, w, c);
  const SideLimiterPartials limiter(g, nu, w[0], w[4], c);
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    double dp, dm;
    side_differences(g, w[k], nb(k, 0), nb(k, 1), nb(k, 2), nb(k, 3), dp, dm);
    up[k] = limited_tape(g, limiter, k, w[k], dp, dm, lj);
  }
}

// upb: the adjoint of the edge state; LJ(i): the taped partials.  Gives the
// adjoints of the interpolants U+ and U- (pu, mu) and adds the face's own
// part to wb.
template <class LjFn>
SPLASH_HD void recon_side_rev(const SideGeom& g, double gam, double dt, const double* w, const double* upb, LjFn LJ,
                              double* pu, double* mu, double* wb) {
  double nub = 0.0;
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    const double dpb = upb[k] * LJ(3 * k), dmb = upb[k] * LJ(3 * k + 1);
    nub = fma(upb[k], LJ(3 * k + 2), nub);
    pu[k] = dpb;
    mu[k] = -dmb;
    wb[k] += upb[k] - dpb + dmb;
  }
  // nu = (c + vn) dt arc / area with c = sqrt(gam Pi / Sigma), vn = -(l . nxr) / Sigma
  const double b = nub * (dt * g.arc_a);
  const double ir = recip(w[0]);
  double ic;
  const double c = root_pair(gam * (w[4] * ir), ic);
  const double vn = -(fdot(g.nxr, d3(w[1], w[2], w[3])) * ir);
  const double cb = (c > 0.0) ? b * 0.5 * ic * gam * ir : 0.0;  // adjoint of Pi, and of Sigma times -Pi / Sigma
  wb[0] -= ir * fma(cb, w[4], b * vn);
  const double s = -b * ir;
  wb[1] = fma(s, g.nxr.x, wb[1]);
  wb[2] = fma(s, g.nxr.y, wb[2]);
  wb[3] = fma(s, g.nxr.z, wb[3]);
  wb[4] += cb;
}

// recon_side_tape for every slot of face f (planes: uplus 5, LJ kTapePlanes)
SPLASH_HD void recon_face_tape(const DevGeom& G, const PhysParams& P, double dt, const double* W, double* uplus,
                               double* LJ, int f) {
  const int fp = G.fpad;
  const int PS = G.max_slots * fp;
  double w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = W[(size_t)k * fp + f];
  const int n = G.nslots[f];
  for (int j = 0; j < n; ++j) {
    const int s = j * fp + f;
    const int st[4] = {G.sten[s], G.sten[PS + s], G.sten[2 * PS + s], G.sten[3 * PS + s]};
    double up[kDim];
    recon_side_tape(
        slot_geom(G, PS, s, n), P.gam, dt, w, [&](int k, int q) { return W[(size_t)k * fp + st[q]]; }, up,
        [&](int i, double x) { LJ[(size_t)i * PS + s] = x; });
#pragma unroll
    for (int k = 0; k < kDim; ++k) uplus[(size_t)k * PS + s] = up[k];
  }
}

// Reverse of recon_face_tape for face f.  W holds the primal (Sigma, l, Pi)
// planes and LJ the slots' tape; upb_at(k, s) returns the adjoint of
// uplus[k * PS + s].  Writes the adjoints of the slot's stencil
// interpolants to PU (planes 0..4: U+, 5..9: U-, each PS long) and adds the
// face's own contribution to wb.  The interpolants' adjoints reach the
// stencil faces through PU times the betas (scattered by the caller).
template <class UpbFn>
SPLASH_HD void recon_face_rev(const DevGeom& G, const PhysParams& P, double dt, const double* W,
                              const double* /*uplus*/, const double* LJ, UpbFn upb_at, double* PU, double* wb, int f) {
  const int fp = G.fpad;
  const int PS = G.max_slots * fp;
  double w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = W[(size_t)k * fp + f];
  const int n = G.nslots[f];
  for (int j = 0; j < n; ++j) {
    const int s = j * fp + f;
    double upb[kDim], pu[kDim], mu[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) upb[k] = upb_at(k, s);
    recon_side_rev(
        slot_geom(G, PS, s, n), P.gam, dt, w, upb, [&](int i) { return LJ[(size_t)i * PS + s]; }, pu, mu, wb);
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      PU[(size_t)k * PS + s] = pu[k];
      PU[(size_t)(kDim + k) * PS + s] = mu[k];
    }
  }
}

// ---------------------------------------------------------------------
// Reverse of the source term.  srcb is the adjoint of res; wb += and
// pb[0..4] += the adjoints of (acc0, omega_acc.y, omega_acc.z, acc_rate,
// total_mass).  omega_acc.x is identically 0 (no derivative taken).
SPLASH_HD void source_rev(const double* w, const D3& fcn, const SrcParams<double>& sp, const PhysParams& P,
                          const double* srcb, double* wb, double* pb) {
  if (!P.accretion_on) return;
  const double b0 = srcb[0], b4 = srcb[4];
  const D3 bl = d3(srcb[1], srcb[2], srcb[3]);
  const double ir = recip(w[0]), ip = recip(w[4]);
  const D3 vel = scal(fcross(fcn, d3(w[1], w[2], w[3])), -ir);
  const double v2 = fdot(vel, vel);
  const D3 omxr = fcross(sp.omega_acc, fcn);
  const D3 rxo = fcross(fcn, omxr);
  const D3 d = sub(omxr, vel);
  const double H = fma(P.gam_gm1 * w[4], ir, 0.5 * v2);
  double w0b = 0.0, w4b = 0.0, v2b = 0.0, gb = 0.0, Hb = 0.0, irb = 0.0;
  // accretion: acc0 (1, r x (omega x r), e_acc + |omega x r - v|^2 / 2)
  pb[0] += fma(b4, fma(0.5, fdot(d, d), P.e_acc), b0 + fdot(bl, rxo));
  const D3 db = scal(d, b4 * sp.acc0);
  D3 ob = fcross(scal(bl, sp.acc0), fcn);
  add_scaled(ob, db, 1.0);
  const D3 omb = fcross(fcn, ob);
  pb[1] += omb.y;
  pb[2] += omb.z;
  D3 velb = scal(db, -1.0);
  if (!P.friction_on) {
    const D3 rxv = fcross(fcn, vel);
    const double im = recip(sp.total_mass);
    const double q = -(sp.acc_rate * (4 * M_PI)) * im, m = q * w[0];
    const double mb = fma(b4, H, b0 + fdot(bl, rxv));
    Hb = b4 * m;
    const D3 x = fcross(scal(bl, m), fcn);
    add_scaled(velb, x, 1.0);
    w0b = mb * q;
    const double qb = mb * w[0];
    pb[3] += qb * (-4 * M_PI) * im;
    pb[4] -= qb * q * im;
  }
  // cooling: - g_eff / kappa (1 - beta(C))
  const double GM = 0.217909;
  const double g_eff = GM - v2;
  const double kappa = 3.4e6;
  const double C = (12. / 5 * 1.6e-13) * (w[0] * ip) * root(root((3. / 4 * 4.85e36) * (g_eff * w[0])));
  const double C_switch = -1 - 1 / (0.736194670678821 - 1);
  double beta, dbeta;
  if (C <= C_switch) {
    const double y = recip(1.0 + C);
    beta = 1.0 - y;
    dbeta = y * y;
  } else {
    const double y = recip(C), x2 = 4.0 * (y * y);
    beta = 1.0 - x2 * x2;
    dbeta = 4.0 * (x2 * x2) * y;
  }
  const bool floor = beta < 1e-8 || is_nan(beta), ceil = beta > 1 - 1e-8;
  if (floor) beta = 1e-8;
  if (ceil) beta = 1 - 1e-8;
  gb = -b4 * (1 / kappa) * (1.0 - beta);
  if (!floor && !ceil && C > 0.0) {
    const double Cb = b4 * g_eff * (1 / kappa) * dbeta * C;  // adjoint of log C
    w0b = fma(1.25 * Cb, ir, w0b);
    w4b = -Cb * ip;
    gb = fma(0.25 * Cb, recip(g_eff), gb);
  }
  if (P.friction_on) {
    const D3 l = d3(w[1], w[2], w[3]);
    const double rho = P.fric_k * g_eff * w[0] * w[0] * ip;
    const D3 vel0 = d3(-P.omega_ns * fcn.y, P.omega_ns * fcn.x, 0.0);
    const D3 rel = sub(vel, vel0);
    double in;
    const double n = root_pair(fdot(rel, rel), in);
    const double k = P.alpha * rho * n;
    D3 wrb = fcross(bl, fcn);
    add_scaled(wrb, vel0, b4);
    const double krb = -fdot(bl, l);
    const double kb = fma(krb, ir, -fma(b4, H, b0 + fdot(wrb, rel)));
    irb = krb * k;
    const double kr = k * ir;
    wb[1] = fma(-kr, bl.x, wb[1]);
    wb[2] = fma(-kr, bl.y, wb[2]);
    wb[3] = fma(-kr, bl.z, wb[3]);
    Hb -= b4 * k;
    add_scaled(velb, wrb, -k);
    if (n > 0.0) add_scaled(velb, rel, kb * P.alpha * rho * in);
    const double rhob = kb * P.alpha * n;
    gb = fma(rhob, P.fric_k * w[0] * w[0] * ip, gb);
    w0b = fma(2.0 * rhob * rho, ir, w0b);
    w4b = fma(-rhob * rho, ip, w4b);
  }
  // H = gam / (gam - 1) Pi / Sigma + v2 / 2, g_eff = GM - v2
  w4b = fma(Hb * P.gam_gm1, ir, w4b);
  irb = fma(Hb * P.gam_gm1, w[4], irb);
  v2b = fma(0.5, Hb, -gb);
  add_scaled(velb, vel, 2.0 * v2b);
  // vel = -(r x l) / Sigma
  w0b -= ir * fma(irb, ir, fdot(velb, vel));
  const D3 lb = fcross(scal(velb, -ir), fcn);
  wb[0] += w0b;
  wb[1] += lb.x;
  wb[2] += lb.y;
  wb[3] += lb.z;
  wb[4] += w4b;
}

// Reverse of prim_of: ub += J^T wb for w = (u0..u3, pressure_fc(u)).
SPLASH_HD void prim_rev(const double* u, const D3& r, double gam, const double* wb, double* ub) {
  const D3 c = fcross(r, d3(u[1], u[2], u[3]));
  const double ir = recip(u[0]), h = 0.5 * fdot(c, c);
  // the floored pressure is a constant
  const double b = less(1e-16, fma(-h, ir, u[4]) * (gam - 1)) ? wb[4] * (gam - 1) : 0.0;
  const D3 lb = fcross(scal(c, -b * ir), r);
  ub[0] += fma(b * h, ir * ir, wb[0]);
  ub[1] += wb[1] + lb.x;
  ub[2] += wb[2] + lb.y;
  ub[3] += wb[3] + lb.z;
  ub[4] += b;
}

}  // namespace rev
}  // namespace f64
}  // namespace splash
