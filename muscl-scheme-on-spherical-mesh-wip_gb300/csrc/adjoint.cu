// Tangent-linear model, forward recomputation and discrete adjoint of the
// FP64 MUSCL step (launchers declared in adjoint.hpp).
//
// Compiled with -fmad=false like step_fp64.cu: the TLM and the
// recomputation run the same per-face bodies (step_body_fp64.cuh), so their
// primal values are bit-identical to the FP64 time step and every branch
// (limiter cases, Riemann sides, HLLC+ switches, floors) is the one the
// forward run took.  The reverse kernels recompute their local primal and
// apply the hand-written reverses of adjoint_rev.cuh.
//
// Reverse of one step (adjoint.hpp gives the forward map), per stage:
//   adj_edge    per edge: la = mask(lam) of its two faces, the adjoint of the
//               edge's flux Fb = dt (coef_1 la_1 - coef_0 la_0), its reverse
//               (dF/duL)^T Fb, (dF/duR)^T Fb; per side: reverse reconstruction
//               from the recomputation's limiter tape -> the adjoints PU of the
//               two interpolants and the side's own part
//   adj_face    per face: lamW = sum over the inverse stencil of beta * PU and
//               the own parts, + source reverse (dt_here la), -> prim reverse
// Every sum has a fixed order (no atomics): the adjoint is deterministic.
//
// The launches overlap by programmatic dependent launch (pdl.cuh), so what a
// predecessor writes is read with ordinary loads: no __restrict__ on those
// pointers, which would let the compiler take the non-coherent path.
// Like the step itself (step_fp64.cu) all of it is bound by the FP64 pipe:
// the flux reverse runs once per edge, the reconstruction on a thread per
// side (forward and tangent: per field of a side on small meshes).
#include <cuda_runtime.h>

#include <cstdint>

#include "adjoint.hpp"
#include "adjoint_rev.cuh"
#include "dual.cuh"
#include "kernels.hpp"
#include "pdl.cuh"
#include "physics_fp64.cuh"
#include "step_body_fp64.cuh"
#include "step_fold_fp64.cuh"
#include "taped.cuh"

namespace splash {
namespace f64 {
// state planes read and written as Taped values (taped.cuh)
template <>
struct Planes<Taped> {
  double* p;
  __device__ Taped ld(size_t i) const { return Taped(p[i]); }
  __device__ void st(size_t i, const Taped& x) const { p[i] = x.v; }
};
}  // namespace f64
}  // namespace splash

namespace splash {
namespace adj {
namespace {

using namespace splash::f64;
using D1 = Dual<1>;
static_assert(kTapeJ == rev::kTapePlanes, "tape plane count");
constexpr int kBlock = 64;                // faces per block
constexpr int kThreads = 2 * kEdgeBlock;  // edge launches: a thread per side, as in step_fp64.cu
inline int edge_blocks(int n) { return (n + kEdgeBlock - 1) / kEdgeBlock; }
// Edge launches with a thread per field of a side up to kPartsEdges edges, at
// two blocks per SM where one for each of the 152 SMs is not enough.  20 steps,
// one thread per side / kDim: tangent on hex(3) 2.20 / 1.70 ms, hex(4) 3.29 /
// 1.97 (one block per SM 2.43), quad(5) 4.45 / 3.32; gradient on hex(3) 3.52 /
// 3.20, quad(4) 4.10 / 3.98 (two blocks per SM, 96 registers: 4.66), hex(4)
// 4.39 / 4.20, quad(5) 7.0 / 6.4.
constexpr int kPartsEdges = 12288;
enum class Split { kSides, kFields, kFieldsTwo };
inline Split edge_split(int n_edges) {
  return n_edges > kPartsEdges ? Split::kSides : edge_blocks(n_edges) > 152 ? Split::kFieldsTwo : Split::kFields;
}

inline int blocks_for(int n) { return (n + kBlock - 1) / kBlock; }
inline int face_blocks(int n) { return (n + kFaces - 1) / kFaces; }

__device__ __forceinline__ D1 dual1(double v, double d) {
  D1 r(v);
  r.d[0] = d;
  return r;
}

// ---------------------------------------------------------------------
// tangent-linear model
__global__ void __launch_bounds__(kBlock) tlm_prepare_kernel(DevGeom G, DevState S, TlmTangents T, PhysParams P) {
  griddep_launch_dependents();
  griddep_wait();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  double vel2 = 0.0, rate2 = 0.0;
  bool negative = false;
  if (f < G.n_faces) {
    const int fp = G.fpad;
    const Planes<D1> U{S.U, T.dU, 0}, W{S.W0, T.dW0, 0};
    D1 u[kDim], w[kDim];
    double wv[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) u[k] = U.ld((size_t)k * fp + f);
    const D3 r = plane3(G.fcn, fp, f);
    prim_of(u, r, P.gam, w);
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      W.st((size_t)k * fp + f, w[k]);
      wv[k] = w[k].v;
    }
    dt_fold(wv, r, P, vel2, rate2, negative);
  }
  fold_warp(vel2, rate2, negative, S, P, gridDim.x * (kBlock / 32));
}

// the flux of edge e, whose sides are columns i and kEdgeBlock + i
__device__ __forceinline__ void tlm_flux(const DevGeom& G, const DevState& S, const TlmTangents& T,
                                         const PhysParams& P, const Gas& gas, const SideExchange<D1, kThreads>& sides,
                                         int e, int i) {
  D1 L[kDim], R[kDim], F[kDim];
  EdgeSide<D1> SL, SR;
  sides.get(i, L, SL);
  sides.get(kEdgeBlock + i, R, SR);
  unsigned bits = riemann_flux(L, R, SL, SR, edge_geom(G, e), gas, P.solver, F);
  const Planes<D1> fe{S.fe, T.dfe, 0};
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    if (nan_bits(F[k].v)) bits |= 1u;
    fe.st((size_t)k * G.epad + e, F[k]);
  }
  if (bits) atomicOr(S.err, bits);
}

template <int STAGE>
__global__ void __launch_bounds__(kThreads, 7) tlm_edge_kernel(DevGeom G, DevState S, TlmTangents T, PhysParams P,
                                                            double dt0) {
  griddep_launch_dependents();
  __shared__ SideExchange<D1, kThreads> sides;
  const Gas gas = gas_of(P);
  const int t = threadIdx.x, i = t & (kEdgeBlock - 1);
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  if (live) {
    const int x = (t < kEdgeBlock) ? e : G.epad + e;
    const SideGeom g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[G.xs + x], G.e_sten[2 * G.xs + x], G.e_sten[3 * G.xs + x]};
    griddep_wait();
    const double dt = (STAGE == 1) ? step_dt(S.scal, dt0) : S.scal[kScDt];
    const Planes<D1> W = (STAGE == 1) ? Planes<D1>{S.W0, T.dW0, 0} : Planes<D1>{S.W1, T.dW1, 0};
    const size_t fp = G.fpad;
    D1 w[kDim], u[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) w[k] = W.ld(k * fp + f);
    recon_side(g, P.gam, dt, w, [&](int k, int q) { return W.ld(k * fp + st[q]); }, u);
    if (STAGE == 1 && x == 0) publish_dt(S, dt);
    sides.put(t, u, edge_side(u, edge_geom(G, e), gas));
  }
  __syncthreads();
  if (!live || t >= kEdgeBlock) return;
  tlm_flux(G, S, T, P, gas, sides, e, i);
}

// with a thread per field of a side, as edge_parts_kernel of step_fp64.cu
template <int STAGE, int BLOCKS>
__global__ void __launch_bounds__(kEdgePartThreads, BLOCKS) tlm_edge_parts_kernel(DevGeom G, DevState S, TlmTangents T,
                                                                          PhysParams P, double dt0) {
  griddep_launch_dependents();
  __shared__ SideExchange<D1, kThreads> sides;
  __shared__ double up[2][kDim][kThreads], nus[2][kThreads];
  __shared__ __align__(8) unsigned char limiters[kThreads * sizeof(SideLimiterPartials)];
  const int warp = threadIdx.x / 32, k = warp >> 1, i = threadIdx.x & 31;
  const int t = (warp & 1) * kEdgeBlock + i;
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const int x = (t < kEdgeBlock) ? e : G.epad + e;
  const size_t fp = G.fpad, xs = G.xs;
  SideLimiterPartials& limiter = reinterpret_cast<SideLimiterPartials*>(limiters)[t];
  SideGeom g{};
  D1 wk, dp, num, dpg;
  if (live) {
    g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    griddep_wait();
    const Planes<D1> W = (STAGE == 1) ? Planes<D1>{S.W0, T.dW0, 0} : Planes<D1>{S.W1, T.dW1, 0};
    wk = W.ld(k * fp + f);
    D1 dm;
    side_differences(g, wk, W.ld(k * fp + st[0]), W.ld(k * fp + st[1]), W.ld(k * fp + st[2]), W.ld(k * fp + st[3]), dp,
                     dm);
    num = dm * g.hr;
    dpg = dp * g.hg;
    if (k == 0) {
      const double dt = (STAGE == 1) ? step_dt(S.scal, dt0) : S.scal[kScDt];
      D1 w[kDim], c;
#pragma unroll
      for (int q = 0; q < kDim; ++q) w[q] = W.ld(q * fp + f);
      const D1 nu = side_courant(g, P.gam, dt, w, c);
      limiter = SideLimiterPartials(g, nu.v, w[0].v, w[4].v, c.v);
      nus[0][t] = nu.v;
      nus[1][t] = nu.d[0];
    } else if (STAGE == 1 && k == kDim - 1 && x == 0) {
      publish_dt(S, step_dt(S.scal, dt0));
    }
  }
  __syncthreads();
  if (live) {
    const D1 u = limited_dual(limiter, k, wk, dp, num, dpg, dual1(nus[0][t], nus[1][t]));
    up[0][k][t] = u.v;
    up[1][k][t] = u.d[0];
  }
  __syncthreads();
  if (k != 0) return;
  const Gas gas = gas_of(P);
  D1 u[kDim];
  if (live) {
#pragma unroll
    for (int q = 0; q < kDim; ++q) u[q] = dual1(up[0][q][t], up[1][q][t]);
    sides.put(t, u, edge_side(u, edge_geom(G, e), gas));
  }
  field0_sync();
  if (!live || t >= kEdgeBlock) return;
  tlm_flux(G, S, T, P, gas, sides, e, i);
}

template <int STAGE>
__global__ void __launch_bounds__(kFaceThreads) tlm_update_kernel(DevGeom G, DevState S, TlmTangents T, PhysParams P) {
  griddep_launch_dependents();
  __shared__ FaceParts<D1, 2 * kDim> parts;
  const int part = face_part(), i = threadIdx.x % kFaces, f = blockIdx.x * kFaces + i;
  const bool live = f < G.n_faces;
  FluxTerms terms;
  if (live && part < kDim) terms = flux_terms(G, f);
  griddep_wait();
  const size_t fp = G.fpad;
  if (live && part < kDim) {
    const Planes<D1> fe{S.fe, T.dfe, 0};
    parts.put(part, i, flux_sum<D1>(G, f, terms, [&](int e) { return fe.ld((size_t)part * G.epad + e); }));
  } else if (live) {
    const SrcParams<D1> sp{dual1(G.acc_src[f], T.dacc[f]),
                           v3(D1(P.omega_acc_x), dual1(P.omega_acc_y, T.d_omega_y), dual1(P.omega_acc_z, T.d_omega_z)),
                           dual1(P.acc_rate, T.d_rate), dual1(P.total_mass, T.d_total_mass)};
    const Planes<D1> Win = (STAGE == 1) ? Planes<D1>{S.W0, T.dW0, 0} : Planes<D1>{S.W1, T.dW1, 0};
    D1 w[kDim], src[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) w[k] = Win.ld(k * fp + f);
    source_term(w, plane3(G.fcn, G.fpad, f), sp, P, src);
#pragma unroll
    for (int k = 0; k < kDim; ++k) parts.put(kDim + k, i, src[k]);
  }
  __syncthreads();
  if (part != 0) return;
  double vel2 = 0.0, rate2 = 0.0;
  bool negative = false;
  if (live) {
    const double dt = S.scal[kScDt];
    const Planes<D1> U{S.U, T.dU, 0};
    D1 sum[kDim], src[kDim], u0[kDim], u[kDim], w[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      sum[k] = parts.get(k, i);
      src[k] = parts.get(kDim + k, i);
      u0[k] = U.ld(k * fp + f);
    }
    bool floored;
    combine_face((STAGE == 1) ? 0.5 * dt : dt, src, sum, u0, u, floored);
    const D3 fcn = plane3(G.fcn, G.fpad, f);
    prim_of(u, fcn, P.gam, w);
    const Planes<D1> Wout = (STAGE == 1) ? Planes<D1>{S.W1, T.dW1, 0} : Planes<D1>{S.W0, T.dW0, 0};
    double wv[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) {
      Wout.st(k * fp + f, w[k]);
      wv[k] = w[k].v;
      if (STAGE == 2) U.st(k * fp + f, u[k]);
    }
    if (STAGE == 2) dt_fold(wv, fcn, P, vel2, rate2, negative);
  }
  if (STAGE == 2) fold_warp(vel2, rate2, negative, S, P, gridDim.x);
}

// ---------------------------------------------------------------------
// branch-frozen forward: the step bodies on Taped (taped.cuh).  A thread per
// face, since a face owns its slice of the tape; it evaluates the fluxes of
// all its edges itself, each in its edge's orientation.
__global__ void __launch_bounds__(kBlock) tp_prim_kernel(DevGeom G, PhysParams P, const double* __restrict__ U,
                                                         double* __restrict__ W) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= G.n_faces) return;
  const int fp = G.fpad;
  Taped u[kDim], w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) u[k] = Taped(U[(size_t)k * fp + f]);
  prim_of(u, plane3(G.fcn, fp, f), P.gam, w);
#pragma unroll
  for (int k = 0; k < kDim; ++k) W[(size_t)k * fp + f] = w[k].v;
}

// the sides of one edge that a face's slot stands for
__device__ __forceinline__ int side_index(const DevGeom& G, int se) {
  return se < 0 ? G.epad + (se & 0x7fffffff) : se;
}

__global__ void __launch_bounds__(kBlock) tp_recon_kernel(DevGeom G, PhysParams P, const double* __restrict__ dtp,
                                                          const double* W, double* uplus) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= G.n_faces) return;
  const size_t fp = G.fpad, xs = G.xs;
  Taped w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = Taped(W[k * fp + f]);
  const int n = G.nslots[f];
  for (int j = 0; j < n; ++j) {
    const int x = side_index(G, G.slot_edge[j * fp + f]);
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    Taped u[kDim];
    recon_side(side_geom(G, x), P.gam, *dtp, w, [&](int k, int q) { return Taped(W[k * fp + st[q]]); }, u);
#pragma unroll
    for (int k = 0; k < kDim; ++k) uplus[k * xs + x] = u[k].v;
  }
}
template <int STAGE>
__global__ void __launch_bounds__(kBlock) tp_flux_kernel(DevGeom G, PhysParams P, const double* __restrict__ dtp,
                                                         const double* Win, const double* U0, const double* uplus,
                                                         double* Uout, double* Wout) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= G.n_faces) return;
  const size_t fp = G.fpad, xs = G.xs;
  const double dt = *dtp;
  Taped u[kDim], w[kDim], u0[kDim], F[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    w[k] = Taped(Win[k * fp + f]);
    u0[k] = Taped(U0[k * fp + f]);
  }
  const Gas gas = gas_of(P);
  Taped src[kDim], sum[kDim];
  source_term(w, plane3(G.fcn, G.fpad, f), face_src_params<double>(G, P, f), P, src);
#pragma unroll
  for (int k = 0; k < kDim; ++k) sum[k] = Taped(0.);
  const int n = G.nslots[f];
  for (int j = 0; j < n; ++j) {
    const int se = G.slot_edge[(size_t)j * fp + f];
    const int e = se & 0x7fffffff;
    Taped L[kDim], R[kDim];
#pragma unroll
    for (int q = 0; q < kDim; ++q) {
      L[q] = Taped(uplus[q * xs + e]);
      R[q] = Taped(uplus[q * xs + (G.e_twin ? G.e_twin[e] : G.epad + e)]);
    }
    riemann_flux(L, R, edge_geom(G, e), gas, P.solver, F);
    const double c = G.e_side[kSideCoef * xs + side_index(G, se)];
#pragma unroll
    for (int k = 0; k < kDim; ++k) sum[k] = fm((se < 0) ? c : -c, F[k], sum[k]);  // flux_sum
  }
  bool floored;
  combine_face((STAGE == 1) ? 0.5 * dt : dt, src, sum, u0, u, floored);
  prim_of(u, plane3(G.fcn, G.fpad, f), P.gam, w);
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    Uout[k * fp + f] = u[k].v;
    Wout[k * fp + f] = w[k].v;
  }
}

// ---------------------------------------------------------------------
// recomputation (double, extra outputs)
__global__ void __launch_bounds__(kBlock) rc_prim_kernel(DevGeom G, PhysParams P, const double* U,
                                                         double* W) {
  griddep_launch_dependents();
  griddep_wait();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= G.n_faces) return;
  const int fp = G.fpad;
  double u[kDim], w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) u[k] = U[(size_t)k * fp + f];
  prim_of(u, plane3(G.fcn, fp, f), P.gam, w);
#pragma unroll
  for (int k = 0; k < kDim; ++k) W[(size_t)k * fp + f] = w[k];
}

__device__ __forceinline__ void rc_flux(const DevGeom& G, const PhysParams& P, const Gas& gas,
                                        const SideExchange<double, kThreads>& sides, double* fe, int e, int i) {
  double L[kDim], R[kDim], F[kDim];
  EdgeSide<double> SL, SR;
  sides.get(i, L, SL);
  sides.get(kEdgeBlock + i, R, SR);
  riemann_flux(L, R, SL, SR, edge_geom(G, e), gas, P.solver, F);
#pragma unroll
  for (int k = 0; k < kDim; ++k) fe[(size_t)k * G.epad + e] = F[k];
}
// the edge launch of the step with the limiter's Jacobian (LJ) and the edge
// states (uplus) kept
__global__ void __launch_bounds__(kThreads) rc_edge_kernel(DevGeom G, PhysParams P, const double* dtp,
                                                           const double* W, double* uplus,
                                                           double* LJ, double* fe) {
  griddep_launch_dependents();
  __shared__ SideExchange<double, kThreads> sides;
  const Gas gas = gas_of(P);
  const int t = threadIdx.x, i = t & (kEdgeBlock - 1);
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  if (live) {
    const int x = (t < kEdgeBlock) ? e : G.epad + e;
    const size_t fp = G.fpad, xs = G.xs;
    const SideGeom g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    griddep_wait();
    double w[kDim], u[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) w[k] = W[k * fp + f];
    rev::recon_side_tape(
        g, P.gam, *dtp, w, [&](int k, int q) { return W[k * fp + st[q]]; }, u,
        [&](int k, double v) { LJ[k * xs + x] = v; });
#pragma unroll
    for (int k = 0; k < kDim; ++k) uplus[k * xs + x] = u[k];
    sides.put(t, u, edge_side(u, edge_geom(G, e), gas));
  }
  __syncthreads();
  if (!live || t >= kEdgeBlock) return;
  rc_flux(G, P, gas, sides, fe, e, i);
}

// with a thread per field of a side
template <int BLOCKS>
__global__ void __launch_bounds__(kEdgePartThreads, BLOCKS) rc_edge_parts_kernel(DevGeom G, PhysParams P, const double* dtp,
                                                                         const double* W, double* uplus, double* LJ,
                                                                         double* fe) {
  griddep_launch_dependents();
  __shared__ SideExchange<double, kThreads> sides;
  __shared__ double up[kDim][kThreads];
  __shared__ __align__(8) unsigned char limiters[kThreads * sizeof(SideLimiterPartials)];
  const int warp = threadIdx.x / 32, k = warp >> 1, i = threadIdx.x & 31;
  const int t = (warp & 1) * kEdgeBlock + i;
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const int x = (t < kEdgeBlock) ? e : G.epad + e;
  const size_t fp = G.fpad, xs = G.xs;
  SideLimiterPartials& limiter = reinterpret_cast<SideLimiterPartials*>(limiters)[t];
  SideGeom g{};
  double wk = 0.0, dp = 0.0, dm = 0.0;
  if (live) {
    g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    griddep_wait();
    const double* Wk = W + k * fp;
    wk = Wk[f];
    side_differences(g, wk, Wk[st[0]], Wk[st[1]], Wk[st[2]], Wk[st[3]], dp, dm);
    if (k == 0) {
      double w[kDim], c;
#pragma unroll
      for (int q = 0; q < kDim; ++q) w[q] = W[q * fp + f];
      const double nu = side_courant(g, P.gam, *dtp, w, c);
      limiter = SideLimiterPartials(g, nu, w[0], w[4], c);
    }
  }
  __syncthreads();
  if (live) {
    const double u = rev::limited_tape(g, limiter, k, wk, dp, dm, [&](int q, double v) { LJ[q * xs + x] = v; });
    up[k][t] = u;
    uplus[k * xs + x] = u;
  }
  __syncthreads();
  if (k != 0) return;
  const Gas gas = gas_of(P);
  double u[kDim];
  if (live) {
#pragma unroll
    for (int q = 0; q < kDim; ++q) u[q] = up[q][t];
    sides.put(t, u, edge_side(u, edge_geom(G, e), gas));
  }
  field0_sync();
  if (!live || t >= kEdgeBlock) return;
  rc_flux(G, P, gas, sides, fe, e, i);
}

template <int STAGE, int BLOCKS>
__global__ void __launch_bounds__(kFaceThreads, BLOCKS) rc_update_kernel(DevGeom G, PhysParams P, const double* dtp,
                                                                 const double* Win,
                                                                 const double* U0,
                                                                 const double* fe, double* Uout,
                                                                 double* Wout, uint8_t* mask) {
  griddep_launch_dependents();
  __shared__ FaceParts<double, 2 * kDim> parts;
  const int part = face_part(), i = threadIdx.x % kFaces, f = blockIdx.x * kFaces + i;
  const bool live = f < G.n_faces;
  FluxTerms terms;
  if (live && part < kDim) terms = flux_terms(G, f);
  griddep_wait();
  const size_t fp = G.fpad;
  if (live && part < kDim) {
    parts.put(part, i, flux_sum<double>(G, f, terms, [&](int e) { return fe[(size_t)part * G.epad + e]; }));
  } else if (live) {
    double w[kDim], src[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) w[k] = Win[k * fp + f];
    source_term(w, plane3(G.fcn, G.fpad, f), face_src_params<double>(G, P, f), P, src);
#pragma unroll
    for (int k = 0; k < kDim; ++k) parts.put(kDim + k, i, src[k]);
  }
  __syncthreads();
  if (part != 0 || !live) return;
  const double dt = *dtp;
  double sum[kDim], src[kDim], u0[kDim], u[kDim], w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    sum[k] = parts.get(k, i);
    src[k] = parts.get(kDim + k, i);
    u0[k] = U0[k * fp + f];
  }
  bool floored;
  combine_face((STAGE == 1) ? 0.5 * dt : dt, src, sum, u0, u, floored);
  prim_of(u, plane3(G.fcn, G.fpad, f), P.gam, w);
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    Uout[k * fp + f] = u[k];
    Wout[k * fp + f] = w[k];
  }
  const uint8_t bit = floored ? (uint8_t)STAGE : (uint8_t)0;
  mask[f] = (STAGE == 1) ? bit : (uint8_t)(mask[f] | bit);
}

// ---------------------------------------------------------------------
// reverse sweep

// lam of face f with the density floor's mask: where the floor held, the
// output's Sigma is a constant
__device__ __forceinline__ double masked(const double* lam, const uint8_t* mask, int bit, size_t fp, int k, int f) {
  return (k == 0 && (mask[f] & bit)) ? 0.0 : lam[k * fp + f];
}

__global__ void __launch_bounds__(kThreads, 7) adj_edge_kernel(DevGeom G, PhysParams P, double dt, double dt_here,
                                                            const double* W,
                                                            const double* uplus,
                                                            const double* LJ,
                                                            const double* lam,
                                                            const uint8_t* mask, int bit,
                                                            double* PU, double* own) {
  griddep_launch_dependents();
  griddep_wait();
  __shared__ SideExchange<double, kThreads> sides;
  __shared__ double bars[rev::kSideBarValues][kThreads];
  const int t = threadIdx.x, i = t & (kEdgeBlock - 1);
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const size_t fp = G.fpad, xs = G.xs;
  const Gas gas = gas_of(P);
  const int x = (t < kEdgeBlock) ? e : G.epad + e;
  EdgeGeom eg;
  EdgeSide<double> S;
  double u[kDim];
  if (live) {
    eg = edge_geom(G, e);
#pragma unroll
    for (int k = 0; k < kDim; ++k) u[k] = uplus[k * xs + x];
    S = edge_side(u, eg, gas);
    sides.put(t, u, S);
  }
  __syncthreads();
  if (live && t < kEdgeBlock) {
    const double* coef = G.e_side + kSideCoef * xs + e;
    const double c0 = dt_here * coef[0], c1 = dt_here * coef[G.epad];
    const int f0 = G.e_face[e], f1 = G.e_face[G.epad + e];
    double R[kDim], Fb[kDim];
    EdgeSide<double> SR;
    sides.get(kEdgeBlock + i, R, SR);
#pragma unroll
    for (int k = 0; k < kDim; ++k)
      Fb[k] = fma(c1, masked(lam, mask, bit, fp, k, f1), -(c0 * masked(lam, mask, bit, fp, k, f0)));
    rev::SideBar BL, BR;
    rev::riemann_flux_rev(u, R, S, SR, eg, gas, P.solver, Fb, BL, BR);
    rev::put_bar(&bars[0][i], kThreads, BL);
    rev::put_bar(&bars[0][kEdgeBlock + i], kThreads, BR);
  }
  __syncthreads();
  if (!live) return;
  const int f = G.e_face[x];
  double w[kDim], upb[kDim] = {0, 0, 0, 0, 0}, pu[kDim], mu[kDim], wb[kDim] = {0, 0, 0, 0, 0};
  rev::SideBar B = rev::get_bar(&bars[0][t], kThreads);
  rev::edge_side_rev(u, S, eg, gas, B, upb);
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = W[k * fp + f];
  rev::recon_side_rev(side_geom(G, x), P.gam, dt, w, upb, [&](int k) { return LJ[k * xs + x]; }, pu, mu, wb);
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    PU[k * xs + x] = pu[k];
    PU[(kDim + k) * xs + x] = mu[k];
    own[k * xs + x] = wb[k];
  }
}

// Four blocks per SM (80 registers instead of 108): the gathers of the five
// field warps wait on memory, and three blocks cover less of it.  20 steps'
// gradient on hex(4) 4.65 -> 4.34 ms, hex(5) 6.99 -> 6.77, hex(6) 21.1 -> 20.4.
template <int STAGE>
__global__ void __launch_bounds__(kFaceThreads, 4) adj_face_kernel(DevGeom G, PhysParams P, double dt_here, AdjScratch X,
                                                                const double* Win,
                                                                const double* Uin,
                                                                const uint8_t* mask, const double* lam,
                                                                double* lam_out) {
  griddep_launch_dependents();
  griddep_wait();
  __shared__ FaceParts<double, 2 * kDim> parts;
  const int part = face_part(), i = threadIdx.x % kFaces, g = blockIdx.x * kFaces + i;
  const bool live = g < G.n_faces;
  const size_t fp = G.fpad, xs = G.xs;
  // the adjoint of this stage's output state: stage 2's is lam, stage 1's lam1
  const double* out = (STAGE == 2) ? lam : X.lam1;
  if (live && part < kDim) {
    // one field over the interpolants whose stencils hold face g, and the
    // sides that are its own
    const double *own = X.own + part * xs, *pu = X.PU + part * xs, *mu = X.PU + (kDim + part) * xs;
    double s = 0.0;
    const int end = X.inv_off[g + 1];
#pragma unroll 4
    for (int e = X.inv_off[g]; e < end; ++e) {
      const int code = X.inv_ent[e];
      const size_t x = (size_t)(code >> 3);
      const int pos = code & 7;
      const double bt = (pos == 4) ? 1.0 : G.e_side[(size_t)(kSideBeta + (pos & 3)) * xs + x];
      s = fma(bt, (pos == 4 ? own : pos >= 2 ? mu : pu)[x], s);
    }
    parts.put(part, i, s);
  } else if (live) {
    double w[kDim], srcb[kDim], wb[kDim] = {0, 0, 0, 0, 0}, pb[5] = {0, 0, 0, 0, 0};
    if (P.accretion_on) {
#pragma unroll
      for (int k = 0; k < kDim; ++k) {
        w[k] = Win[k * fp + g];
        srcb[k] = dt_here * masked(out, mask, STAGE, fp, k, g);
      }
      rev::source_rev(w, plane3(G.fcn, G.fpad, g), face_src_params<double>(G, P, g), P, srcb, wb, pb);
#pragma unroll
      for (int j = 0; j < 5; ++j) X.th[j * fp + g] += pb[j];
    }
#pragma unroll
    for (int k = 0; k < kDim; ++k) parts.put(kDim + k, i, wb[k]);
  }
  __syncthreads();
  if (part != 0 || !live) return;
  double wb[kDim], u[kDim], ub[kDim] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    wb[k] = parts.get(k, i) + parts.get(kDim + k, i);
    u[k] = Uin[k * fp + g];
  }
  rev::prim_rev(u, plane3(G.fcn, G.fpad, g), P.gam, wb, ub);
  if (STAGE == 2) {
#pragma unroll
    for (int k = 0; k < kDim; ++k) lam_out[k * fp + g] = ub[k];
  } else {
    // U1 = floor(U + acc1) and U2 = floor(U + acc2) both hold U directly
#pragma unroll
    for (int k = 0; k < kDim; ++k)
      lam_out[k * fp + g] = ub[k] + masked(out, mask, 1, fp, k, g) + masked(lam, mask, 2, fp, k, g);
  }
}

}  // namespace
}  // namespace adj

// ---- launchers ----------------------------------------------------------
cudaError_t tlm_prepare(const DevGeom& G, const DevState& S, const TlmTangents& T, const PhysParams& P,
                        cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(S.fold, 0, kFoldCount * sizeof(*S.fold), st);
  if (e != cudaSuccess) return e;
  adj::tlm_prepare_kernel<<<adj::blocks_for(G.n_faces), adj::kBlock, 0, st>>>(G, S, T, P);
  return cudaGetLastError();
}

cudaError_t tlm_step(const DevGeom& G, const DevState& S, const TlmTangents& T, const PhysParams& P, double dt0,
                     cudaStream_t st) {
  FirstError chk;
  const int nb = adj::face_blocks(G.n_faces), ne = adj::edge_blocks(G.n_edges);
  const adj::Split split = adj::edge_split(G.n_edges);
  const dim3 eb(split == adj::Split::kSides ? adj::kThreads : f64::kEdgePartThreads);
  using Edge = void (*)(DevGeom, DevState, TlmTangents, PhysParams, double);
  const Edge edge1 = split == adj::Split::kSides    ? adj::tlm_edge_kernel<1>
                     : split == adj::Split::kFields ? adj::tlm_edge_parts_kernel<1, 1>
                                                    : adj::tlm_edge_parts_kernel<1, 2>;
  const Edge edge2 = split == adj::Split::kSides    ? adj::tlm_edge_kernel<2>
                     : split == adj::Split::kFields ? adj::tlm_edge_parts_kernel<2, 1>
                                                    : adj::tlm_edge_parts_kernel<2, 2>;
  chk(launch_pdl(edge1, dim3(ne), eb, st, G, S, T, P, dt0));
  chk(launch_pdl(adj::tlm_update_kernel<1>, dim3(nb), dim3(f64::kFaceThreads), st, G, S, T, P));
  chk(launch_pdl(edge2, dim3(ne), eb, st, G, S, T, P, dt0));
  chk(launch_pdl(adj::tlm_update_kernel<2>, dim3(nb), dim3(f64::kFaceThreads), st, G, S, T, P));
  return chk.status();
}

namespace {
// points the comparisons of the next launch at its tape region (the
// __constant__ update is ordered on the stream before the launch) and
// restarts every face's position
cudaError_t tape_region(const DevGeom& G, uint32_t* region, uint32_t* pos, unsigned* err, int mode,
                        cudaStream_t st) {
  // err[2..3] hold the 64-bit flip count
  const tape::TapeCfg cfg{region, pos, err, reinterpret_cast<unsigned long long*>(err + 2), mode};
  cudaError_t e = cudaMemcpyToSymbolAsync(tape::g_tape, &cfg, sizeof cfg, 0, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  return cudaMemsetAsync(pos, 0, (size_t)G.n_faces * sizeof(uint32_t), st);
}
}  // namespace

int taped_words_per_face() { return tape::kTapeWords; }

cudaError_t taped_prim(const DevGeom& G, const PhysParams& P, double* U, double* W, uint32_t* region,
                       uint32_t* pos, unsigned* err, int mode, cudaStream_t st) {
  cudaError_t e = tape_region(G, region, pos, err, mode, st);
  if (e != cudaSuccess) return e;
  adj::tp_prim_kernel<<<adj::blocks_for(G.n_faces), adj::kBlock, 0, st>>>(G, P, U, W);
  return cudaGetLastError();
}

cudaError_t taped_step(const DevGeom& G, const PhysParams& P, const double* dtp, double* U, double* W0,
                       double* W1, double* uplus, double* U1, uint32_t* region, uint32_t* pos, unsigned* err,
                       int mode, cudaStream_t st) {
  const int nb = adj::blocks_for(G.n_faces);
  constexpr int B = adj::kBlock;
  const size_t RW = (size_t)G.n_faces * tape::kTapeWords;
  cudaError_t e;
  if ((e = tape_region(G, region, pos, err, mode, st)) != cudaSuccess) return e;
  adj::tp_recon_kernel<<<nb, B, 0, st>>>(G, P, dtp, W0, uplus);
  if ((e = tape_region(G, region + RW, pos, err, mode, st)) != cudaSuccess) return e;
  adj::tp_flux_kernel<1><<<nb, B, 0, st>>>(G, P, dtp, W0, U, uplus, U1, W1);
  if ((e = tape_region(G, region + 2 * RW, pos, err, mode, st)) != cudaSuccess) return e;
  adj::tp_recon_kernel<<<nb, B, 0, st>>>(G, P, dtp, W1, uplus);
  if ((e = tape_region(G, region + 3 * RW, pos, err, mode, st)) != cudaSuccess) return e;
  adj::tp_flux_kernel<2><<<nb, B, 0, st>>>(G, P, dtp, W1, U, uplus, U, W0);
  return cudaGetLastError();
}

cudaError_t rc_prim(const DevGeom& G, const PhysParams& P, const double* U, double* W, cudaStream_t st) {
  adj::rc_prim_kernel<<<adj::blocks_for(G.n_faces), adj::kBlock, 0, st>>>(G, P, U, W);
  return cudaGetLastError();
}

cudaError_t rc_step(const DevGeom& G, const PhysParams& P, const double* dtp, const StepTape& t, double* fe,
                    double* U_next, double* W_next, cudaStream_t st) {
  FirstError chk;
  const int nb = adj::face_blocks(G.n_faces), ne = adj::edge_blocks(G.n_edges);
  constexpr int B = f64::kFaceThreads;
  const bool five = f64::five_face_blocks(G.n_faces);
  const adj::Split split = adj::edge_split(G.n_edges);
  const dim3 eb(split == adj::Split::kSides ? adj::kThreads : f64::kEdgePartThreads);
  using Edge = void (*)(DevGeom, PhysParams, const double*, const double*, double*, double*, double*);
  const Edge edge = split == adj::Split::kSides    ? adj::rc_edge_kernel
                    : split == adj::Split::kFields ? adj::rc_edge_parts_kernel<1>
                                                   : adj::rc_edge_parts_kernel<2>;
  chk(launch_pdl(edge, dim3(ne), eb, st, G, P, dtp, t.W0, t.P0, t.J0, fe));
  chk(launch_pdl(five ? adj::rc_update_kernel<1, 5> : adj::rc_update_kernel<1, 4>, dim3(nb), dim3(B), st, G, P, dtp, t.W0, t.U, fe, t.U1, t.W1, t.mask));
  chk(launch_pdl(edge, dim3(ne), eb, st, G, P, dtp, t.W1, t.P1, t.J1, fe));
  chk(launch_pdl(five ? adj::rc_update_kernel<2, 5> : adj::rc_update_kernel<2, 4>, dim3(nb), dim3(B), st, G, P, dtp, t.W1, t.U, fe, U_next, W_next, t.mask));
  return chk.status();
}

cudaError_t adj_step(const DevGeom& G, const PhysParams& P, double dt, const StepTape& t, const AdjScratch& X,
                     double* lam, cudaStream_t st) {
  FirstError chk;
  const int nb = adj::face_blocks(G.n_faces), ne = adj::edge_blocks(G.n_edges);
  constexpr int B = f64::kFaceThreads, E = adj::kThreads;
  // stage 2: U2 = floor(U + dt Phi(W1, P1))
  chk(launch_pdl(adj::adj_edge_kernel, dim3(ne), dim3(E), st, G, P, dt, dt, t.W1, t.P1, t.J1, lam, t.mask, 2, X.PU, X.own));
  chk(launch_pdl(adj::adj_face_kernel<2>, dim3(nb), dim3(B), st, G, P, dt, X, t.W1, t.U1, t.mask, lam, X.lam1));
  // stage 1: U1 = floor(U + dt/2 Phi(W0, P0))
  const double dt_half = dt / 2;
  chk(launch_pdl(adj::adj_edge_kernel, dim3(ne), dim3(E), st, G, P, dt, dt_half, t.W0, t.P0, t.J0, X.lam1, t.mask, 1, X.PU, X.own));
  chk(launch_pdl(adj::adj_face_kernel<1>, dim3(nb), dim3(B), st, G, P, dt_half, X, t.W0, t.U, t.mask, lam, lam));
  return chk.status();
}

}  // namespace splash
