// Per-face bodies of the FP64 MUSCL step, shared by the time step
// (step_fp64.cu, scalar type double), the tangent-linear model (Dual<N>)
// and the adjoint's forward recomputation (double, extra outputs).
//
// Every body evaluates one face or one side of an edge
// (MUSCL_base.hpp:124-161, 238-276, 345-434, 517-562), so all users of a
// body produce bit-identical primal values when compiled with -fmad=false.
#pragma once

#include <cstddef>

#include "dual.cuh"
#include "layout.hpp"
#include "limiter_pair.cuh"
#include "physics_fp64.cuh"

namespace splash {
namespace f64 {

// A set of planes of doubles (value) and, for Dual<N>, N tangent copies
// of the same layout `tstride` doubles apart.
template <class T>
struct Planes;

template <>
struct Planes<double> {
  double* p;
  SPLASH_HD double ld(size_t i) const { return p[i]; }
  SPLASH_HD void st(size_t i, double x) const { p[i] = x; }
};

template <int N>
struct Planes<Dual<N>> {
  double* p;
  double* t;
  size_t tstride;
  SPLASH_HD Dual<N> ld(size_t i) const {
    Dual<N> r(p[i]);
#pragma unroll
    for (int j = 0; j < N; ++j) r.d[j] = t[j * tstride + i];
    return r;
  }
  SPLASH_HD void st(size_t i, const Dual<N>& x) const {
    p[i] = x.v;
#pragma unroll
    for (int j = 0; j < N; ++j) t[j * tstride + i] = x.d[j];
  }
};

SPLASH_HD D3 plane3(const double* p, int stride, int i) {
  return D3{p[i], p[stride + i], p[2 * stride + i]};
}

// (Sigma, l, Pi) of a conserved state u; MUSCL_base.hpp:124-161 stores
// U_i - 0.0 for fields 0..3 and the pressure of MUSCL_base.hpp:517-539.
template <class T>
SPLASH_HD void prim_of(const T* u, const D3& r, double gam, T* w) {
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = u[k] - 0.0;
  w[4] = pressure_fc(u, r, gam) - 0.0;
}

// The accretion parameters of one face, in the scalar type Q.
template <class Q>
SPLASH_HD SrcParams<Q> face_src_params(const DevGeom& G, const PhysParams& P, int f) {
  return SrcParams<Q>{Q(G.acc_src[f]), v3(Q(P.omega_acc_x), Q(P.omega_acc_y), Q(P.omega_acc_z)),
                      Q(P.acc_rate), Q(P.total_mass)};
}

// The constants of one side of an edge (one slot): interpolation weights,
// H+/H-, BM/H+, the limiter's eta_plus and superbee scale eta_minus / (2 N),
// arc / area and cross(normal, edge centre).
struct SideGeom {
  double b0, b1, b2, b3, hr, hg, eta_p, sbs, arc_a;
  D3 nxr;
};
// ... of side x (DevGeom::e_side)
SPLASH_HD SideGeom side_geom(const DevGeom& G, int x) {
  const size_t xs = (size_t)G.xs;
  const double* p = G.e_side + x;
  SideGeom c;
  c.b0 = p[kSideBeta * xs];
  c.b1 = p[(kSideBeta + 1) * xs];
  c.b2 = p[(kSideBeta + 2) * xs];
  c.b3 = p[(kSideBeta + 3) * xs];
  c.hr = p[kSideHr * xs];
  c.hg = p[kSideHg * xs];
  c.eta_p = p[kSideEtaP * xs];
  c.sbs = p[kSideSbs * xs];
  c.arc_a = p[kSideArc * xs];
  c.nxr = D3{p[kSideNxr * xs], p[(kSideNxr + 1) * xs], p[(kSideNxr + 2) * xs]};
  return c;
}
// ... from the slot planes (stride PS), at index s, of a face of n edges
SPLASH_HD SideGeom slot_geom(const DevGeom& G, int PS, int s, int n) {
  SideGeom c;
  c.b0 = G.beta[s];
  c.b1 = G.beta[PS + s];
  c.b2 = G.beta[2 * PS + s];
  c.b3 = G.beta[3 * PS + s];
  c.arc_a = G.arc_a[s];
  c.hr = G.hpm[s] / G.hpm[PS + s];
  c.hg = G.bm[s] / G.hpm[s];
  c.eta_p = G.eta[s];
  c.sbs = G.eta[PS + s] / (2 * n);
  const D3 ec = plane3(G.ec, PS, s), en = plane3(G.en, PS, s);
  const double ecn = G.ecn[s];
  c.nxr = cross3(en, d3(ec.x / ecn, ec.y / ecn, ec.z / ecn));
  return c;
}
// The edge as the flux sees it, in the orientation of side 0
SPLASH_HD EdgeGeom edge_geom(const DevGeom& G, int e) {
  const size_t ep = (size_t)G.epad, xs = (size_t)G.xs;
  const double *p = G.e_geo + e, *q = G.e_side + kSideNxr * xs + e;
  return EdgeGeom{D3{p[0], p[ep], p[2 * ep]}, D3{p[3 * ep], p[4 * ep], p[5 * ep]}, D3{q[0], q[xs], q[2 * xs]}};
}

// Courant factor of the limiter (adiabatic.hpp:741-758, 792-810) of the
// face state w on one side of an edge, (c + v.n) dt arc / area with
// v.n = -(l . (n x R)) / Sigma, and what the limiter makes of it.
template <class T>
SPLASH_HD T side_courant(const SideGeom& g, double gam, double dt, const T* w, T& c) {
  const T ir = recip(w[0]);
  c = root(gam * (w[4] * ir));
  const T vn = -(fdot(g.nxr, v3(w[1], w[2], w[3])) * ir);
  return (c + vn) * (dt * g.arc_a);
}
SPLASH_HD LimiterLine<double> limiter_line(double eta_p, double sbs, double nu) {
  const double ts = fma(nu, 1.0 / 3, 1.0 / 3);
  return LimiterLine<double>{eta_p, divide(sbs, nu), ts, 1.0 - ts};
}

// The differences of one field across the side: dp = U+ - w, dm = w - U-
// with the interpolants U+- at the distances H+- (MUSCL_base.hpp:361-434).
template <class T>
SPLASH_HD void side_differences(const SideGeom& g, const T& w, const T& a, const T& b, const T& c, const T& d, T& dp,
                                T& dm) {
  dp = fm(g.b1, b, fm(g.b0, a, -w));
  dm = fm(-g.b3, d, fm(-g.b2, c, w));
}
// r = num / dp with num = hr dm: (dm / H-) / (dp / H+)
SPLASH_HD double slope_ratio(double dp, double num) {
  const double v = num * recip(dp);
  return odd_bits(v) ? exact_quotient(num, dp) : v;
}

// The limiter of one field in FP64; out of line, as the rarer path.
SPLASH_COLD double limiter_full(double dp, double num, double eta_p, double sb, double ts, double t1) {
  const LimiterLine<double> line{eta_p, sb, ts, t1};
  const bool pos = (int64_t)bits_of(sb) > 0 && !odd_bits(sb);
  const double r = slope_ratio(dp, num);
  return pos ? limiter_field_pos(r, line) : limiter_field(r, line);
}

// One side's limiter: what its fields share, and the value for one field.
struct SideLimiter {
  double eta_p, sbs, nu;
#if defined(SPLASH_SWITCH_TABLE)
  PairLine pairs;
#endif
  int scale[kDim];  // exponent fields that the differences are measured against

  // The differences of Sigma and Pi are measured against the face's own
  // values, those of l against Sigma c: the momentum equation carries Pi =
  // Sigma c^2 / gam beside them.
  SPLASH_HD SideLimiter(const SideGeom& g, double nu_, double w0, double w4, double c)
      : eta_p(g.eta_p), sbs(g.sbs), nu(nu_) {
    scale[0] = exponent_field(w0);
    scale[1] = scale[2] = scale[3] = scale[0] + exponent_field(c) - 1023;
    scale[4] = exponent_field(w4);
#if defined(SPLASH_SWITCH_TABLE)
    pairs = pair_line(eta_p, sbs, nu);
#endif
  }
  // the limiter in pairs of floats, where they serve; dpg = dp BM / H+
  SPLASH_HD bool in_pairs(int k, double dp, double num, double dpg, double& lim) const {
#if defined(SPLASH_SWITCH_TABLE)
    return shallow(dpg, scale[k]) && limiter_pair(dp, num, dp - num, pairs, lim);
#else
    return false;
#endif
  }
  // line: limiter_line of the side, used where pairs do not serve
  SPLASH_HD double operator()(int k, double dp, double num, double dpg, const LimiterLine<double>& line) const {
    double lim;
    if (in_pairs(k, dp, num, dpg, lim)) return lim;
    return limiter_full(dp, num, line.eta_p, line.sb, line.ts, line.t1);
  }
  // whether any field may need the line
  SPLASH_HD bool needs_line(const double* dp, const double* num, const double* dpg) const {
#if defined(SPLASH_SWITCH_TABLE)
    bool need = !pairs.ok;
#pragma unroll
    for (int k = 0; k < kDim; ++k) need = need || !shallow(dpg[k], scale[k]) || !pair_range(dp[k], num[k]);
    return need;
#else
    return true;
#endif
  }
};

// The limiter of one field with its partial derivatives in r and nu.  The
// value is SideLimiter's, bit for bit.
struct Phi {
  double v, r, nu;
};
// known: the switch is h (8 FP64 instructions less).
SPLASH_HD Phi limiter_partials(double r, const LimiterLine<double>& l, double inu, bool known, double hk) {
  if (nan_bits(r)) return Phi{0., 0., 0.};
  if (odd_bits(r)) return Phi{limiter_field(r, l), 0., 0.};  // flat in r and in the Courant factor
  // the superbee: max(0, max(min(1, r sb), min(r, eta_p)))
  Phi A{1., 0., 0.};
  const double rs = r * l.sb;
  if (less(rs, 1.)) A = Phi{rs, l.sb, -rs * inu};
  const Phi B = less(l.eta_p, r) ? Phi{l.eta_p, 0., 0.} : Phi{r, 1., 0.};
  Phi sb = less(A.v, B.v) ? B : A;
  if (!less(0., sb.v)) sb = Phi{0., 0., 0.};
  // the third-order line t1 + ts r below it, not below 0
  const double t = fma(l.ts, r, l.t1);
  Phi to = sb;
  if (less(t, sb.v)) to = Phi{t, l.ts, (r - 1) * (1.0 / 3)};
  if (!less(0., to.v)) to = Phi{0., 0., 0.};
  if (to.v == sb.v) return sb;
  if (!(r > 0.0)) return to;
  double slope;
  const double h = switch_slope(r, known, hk, slope);
  return Phi{fma(h, sb.v - to.v, to.v), fma(h, sb.r - to.r, fma(slope, sb.v - to.v, to.r)),
             fma(h, sb.nu - to.nu, to.nu)};
}
struct SideLimiterPartials : SideLimiter {
  LimiterLine<double> line;
  double inu;
  SPLASH_HD SideLimiterPartials(const SideGeom& g, double nu_, double w0, double w4, double c)
      : SideLimiter(g, nu_, w0, w4, c), line(limiter_line(g.eta_p, g.sbs, nu_)), inu(recip(nu_)) {}
  // r receives the ratio
  SPLASH_HD Phi operator()(int k, double dp, double num, double dpg, double& r) const {
    r = slope_ratio(dp, num);
    // in pairs the switch comes with the value and serves the derivatives
    // too, where it was needed (h > 0)
    bool in_pairs = false, known = false;
    double v = 0.0, hk = 0.0;
#if defined(SPLASH_SWITCH_TABLE)
    Pair h{0.0f, 0.0f};
    in_pairs = shallow(dpg, scale[k]) && limiter_pair(dp, num, dp - num, pairs, v, h);
    known = in_pairs && h.h > 0.0f;
    if (known) hk = widen(h.h) + widen(h.l);
#endif
    Phi phi = limiter_partials(r, line, inu, known, hk);
    if (in_pairs) phi.v = v;
    return phi;
  }
};

// up = w + dpg phi(r, nu) of field k with its tangents
template <int N>
SPLASH_HD Dual<N> limited_dual(const SideLimiterPartials& limiter, int k, const Dual<N>& w, const Dual<N>& dp,
                               const Dual<N>& num, const Dual<N>& dpg, const Dual<N>& nu) {
  double r;
  const Phi phi = limiter(k, dp.v, num.v, dpg.v, r);
  const bool flat = odd_bits(r);  // the limiter is flat where the ratio is no number
  const double idp = flat ? 0.0 : recip(dp.v);
  Dual<N> lim(phi.v);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double rd = flat ? 0.0 : fma(-r, dp.d[i], num.d[i]) * idp;
    lim.d[i] = fma(phi.r, rd, phi.nu * nu.d[i]);
  }
  return fm(dpg, lim, w);
}

// The limited state (Sigma, l, Pi) of one side: up = w + dp phi(r) BM / H+.
// nb(k, q) returns field k of stencil face q (0, 1: plus pair, 2, 3: minus).
template <class T, class NbFn>
SPLASH_HD void recon_side(const SideGeom& g, double gam, double dt, const T* w, NbFn nb, T* up) {
  T c;
  const T nu = side_courant(g, gam, dt, w, c);
  using Limiter = std::conditional_t<is_dual<T>::value, SideLimiterPartials, SideLimiter>;
  const Limiter limiter(g, val(nu), val(w[0]), val(w[4]), val(c));
  T num[kDim], dpg[kDim], dp[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    T dm;
    side_differences(g, w[k], nb(k, 0), nb(k, 1), nb(k, 2), nb(k, 3), dp[k], dm);
    num[k] = dm * g.hr;
    dpg[k] = dp[k] * g.hg;
  }
  if constexpr (is_dual<T>::value) {
#pragma unroll
    for (int k = 0; k < kDim; ++k) up[k] = limited_dual(limiter, k, w[k], dp[k], num[k], dpg[k], nu);
  } else {
    double dpv[kDim], numv[kDim], dpgv[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      dpv[k] = val(dp[k]);
      numv[k] = val(num[k]);
      dpgv[k] = val(dpg[k]);
    }
    LimiterLine<double> line{};
    if (limiter.needs_line(dpv, numv, dpgv)) {
#if defined(__CUDA_ARCH__)
      asm volatile("");  // a branch: evaluated beside it, the line costs 8 FP64 instructions on every path
#endif
      line = limiter_line(g.eta_p, g.sbs, val(nu));
    }
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      T lim;
      if constexpr (std::is_same<T, double>::value) {
        lim = limiter(k, dpv[k], numv[k], dpgv[k], line);
      } else {
        // the recorded branches decide; where they are the values' own, so is the value
        const LimiterLine<double> all = limiter_line(g.eta_p, g.sbs, val(nu));
        const double r = slope_ratio(dpv[k], numv[k]);
        lim = limiter_field(T(r), LimiterLine<T>{all.eta_p, T(all.sb), T(all.ts), T(all.t1)});
        if (bits_of(val(lim)) == bits_of(limiter_field(r, all)))
          lim = T(limiter(k, dpv[k], numv[k], dpgv[k], line));
      }
      up[k] = fm(dpg[k], lim, w[k]);
    }
  }
}

// find_U_edges for every slot of face f from the slot planes: the edge
// states (Sigma, l, Pi)
template <class T>
SPLASH_HD void recon_face(const DevGeom& G, const PhysParams& P, double dt, const Planes<T>& W,
                          const Planes<T>& uplus, int f) {
  const int fp = G.fpad;
  const int PS = G.max_slots * fp;  // one slot-plane set
  T w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = W.ld((size_t)k * fp + f);
  const int n = G.nslots[f];
  for (int j = 0; j < n; ++j) {
    const int s = j * fp + f;
    const int st[4] = {G.sten[s], G.sten[PS + s], G.sten[2 * PS + s], G.sten[3 * PS + s]};
    T up[kDim];
    recon_side(slot_geom(G, PS, s, n), P.gam, dt, w, [&](int k, int q) { return W.ld((size_t)k * fp + st[q]); }, up);
#pragma unroll
    for (int k = 0; k < kDim; ++k) uplus.st((size_t)k * PS + s, up[k]);
  }
}

#if defined(__CUDACC__)
// The edge launches with a thread per field of a side (small meshes): warp
// 2 k + s of a block serves field k of side s of its kEdgeBlock edges.
constexpr int kEdgePartThreads = 2 * kEdgeBlock * kDim;
// the barrier of the two field 0 warps, which go on alone
__device__ __forceinline__ void field0_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

// What the two threads of an edge exchange: each puts the state and the
// EdgeSide of its side, the one that evaluates the flux takes both.  One
// shared-memory plane per value (and one per tangent), indexed by thread.
template <class T, int THREADS>
struct SideExchange {
  static constexpr int kValues = kDim + 10;
  static constexpr int kParts = is_dual<T>::value ? 2 : 1;
  double v[kParts][kValues][THREADS];

  __device__ __forceinline__ void put(int i, int t, const T& x) {
    v[0][i][t] = val(x);
    if constexpr (is_dual<T>::value) v[1][i][t] = x.d[0];
  }
  __device__ __forceinline__ T get(int i, int t) const {
    T x(v[0][i][t]);
    if constexpr (is_dual<T>::value) x.d[0] = v[1][i][t];
    return x;
  }
  __device__ __forceinline__ void put(int t, const T* u, const EdgeSide<T>& S) {
#pragma unroll
    for (int k = 0; k < kDim; ++k) put(k, t, u[k]);
    const T s[10] = {S.vel.x, S.vel.y, S.vel.z, S.vn, S.v2, S.p, S.e, S.gi, S.a2, S.a};
#pragma unroll
    for (int k = 0; k < 10; ++k) put(kDim + k, t, s[k]);
  }
  __device__ __forceinline__ void get(int t, T* u, EdgeSide<T>& S) const {
#pragma unroll
    for (int k = 0; k < kDim; ++k) u[k] = get(k, t);
    T s[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) s[k] = get(kDim + k, t);
    S.vel = v3(s[0], s[1], s[2]);
    S.vn = s[3];
    S.v2 = s[4];
    S.p = s[5];
    S.e = s[6];
    S.gi = s[7];
    S.a2 = s[8];
    S.a = s[9];
  }
};
#endif

// res2d and the RK combine with the density floor (MUSCL_base.hpp:238-276,
// 124-161) of face f, in three parts that the kernels spread over threads:
// the sum over the face's slots of -+ coef flux of one field (flux(e): that
// field of edge e's flux), the source (source_term), and the combination.
// The edges of slots j0 .. j0 + kTerms - 1 of face f and their coefficients
// (negated on the owner side), loaded without waiting for the slot count: the
// planes hold max_slots entries of every face.
constexpr int kTerms = 6;
struct FluxTerms {
  int e[kTerms];
  double c[kTerms];
};
SPLASH_HD FluxTerms flux_terms(const DevGeom& G, int f, int j0 = 0) {
  FluxTerms t;
#pragma unroll
  for (int j = 0; j < kTerms; ++j) {
    const int se = (j0 + j < G.max_slots) ? G.slot_edge[(size_t)(j0 + j) * G.fpad + f] : 0;
    t.e[j] = se & 0x7fffffff;
    const double c = G.e_side[(size_t)kSideCoef * G.xs + (se < 0 ? G.epad + t.e[j] : t.e[j])];
    t.c[j] = (se < 0) ? c : -c;
  }
  return t;
}
// `first` is flux_terms of slot 0; a chunk's fluxes are in flight together
template <class T, class FluxFn>
SPLASH_HD T flux_sum(const DevGeom& G, int f, const FluxTerms& first, FluxFn flux) {
  T acc(0.);
  const int n = G.nslots[f];
  FluxTerms t = first;
  for (int j0 = 0;;) {
    T F[kTerms];
#pragma unroll
    for (int j = 0; j < kTerms; ++j) F[j] = flux(t.e[j]);
#pragma unroll
    for (int j = 0; j < kTerms; ++j)
      if (j0 + j < n) acc = fm(t.c[j], F[j], acc);
    j0 += kTerms;
    if (j0 >= n) return acc;
    t = flux_terms(G, f, j0);
  }
}
// U0 + dt_here (source + sum), floored; `floored` reports the density floor
template <class T>
SPLASH_HD void combine_face(double dt_here, const T* src, const T* sum, const T* u0, T* u, bool& floored) {
#pragma unroll
  for (int k = 0; k < kDim; ++k) u[k] = fm(dt_here, src[k] + sum[k], u0[k]);
  floored = less(u[0], T(1e-8));
  if (floored) u[0] = T(1e-8);
}

#if defined(__CUDACC__)
// A block of the face launches: kFaces faces, and for each of them kDim
// threads that sum one field's fluxes and one for the source, a warp per
// part, so that the parts run side by side on the SM's four schedulers; the
// warp of part 0 then combines them.  One thread per face runs all of it in
// sequence, 194 dependent FP64 instructions of 33 ns on a mesh that leaves
// the SMs a warp or two.  The parts rotate from block to block, since a
// warp's place in the block decides its scheduler and the source is the
// longest part.
constexpr int kFaces = 32;
constexpr int kFaceThreads = kFaces * (kDim + 1);
// Blocks per SM that a face launch of n_faces is compiled for: 5 (64
// registers) where more than the 4 that fit at 66-70 registers are there for
// each of the GB300's 152 SMs.  us per step, 4 / 5: hex(5) 76 / 79, hex(6)
// 230 / 217.
inline bool five_face_blocks(int n_faces) { return (n_faces + kFaces - 1) / kFaces > 4 * 152; }
__device__ __forceinline__ int face_part() { return (int)((threadIdx.x / kFaces + blockIdx.x) % (kDim + 1)); }
template <class T, int N>
struct FaceParts {
  static constexpr int kParts = is_dual<T>::value ? 2 : 1;
  double v[kParts][N][kFaces];
  __device__ __forceinline__ void put(int i, int t, const T& x) {
    v[0][i][t] = val(x);
    if constexpr (is_dual<T>::value) v[1][i][t] = x.d[0];
  }
  __device__ __forceinline__ T get(int i, int t) const {
    T x(v[0][i][t]);
    if constexpr (is_dual<T>::value) x.d[0] = v[1][i][t];
    return x;
  }
};
#endif

}  // namespace f64
}  // namespace splash
