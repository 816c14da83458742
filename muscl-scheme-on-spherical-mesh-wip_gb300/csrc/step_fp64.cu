// FP64 kernels of the MUSCL time step (the reference method in FP64).
//
// One do_step(dt0) (MUSCL_base/MUSCL_base.hpp:97-225) is four launches on
// one stream, captured into a CUDA graph by the host:
//
//   edge(W0)    per edge : dt clip; limited states of both sides, Riemann flux
//   update(1)   per face : source, res2d(dt/2) + U0 -> W1 (Sigma, l, Pi)
//   edge(W1)    per edge
//   update(2)   per face : res2d(dt) + U0 -> U, W0 for the next step, and the
//                          candidates of its dt, folded; the last block makes
//                          the bounds of them
//
// What bounds them is the FP64 pipe (fp64_math.cuh: one warp instruction per
// SM every 8.2 ns), so the layout serves the instruction count: every edge's
// flux is evaluated once (every Riemann solver here satisfies
// F(uR, uL, -n) = -F(uL, uR, n) term by term; the reference evaluates it from
// both faces), and the work is spread over sides and edges instead of faces,
// so that small meshes reach every SM.  Faces sum their edges' fluxes in the
// reference's slot order.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.hpp"
#include "pdl.cuh"
#include "physics_fp64.cuh"
#include "physics_iso.cuh"
#include "step_body_fp64.cuh"
#include "step_fold_fp64.cuh"

namespace splash {
namespace f64 {
namespace {

// Edge launches: blocks of kEdgeBlock edges and twice as many threads.
// Thread t reconstructs one side of edge t mod kEdgeBlock and evaluates what
// the flux needs of that side alone (EdgeSide); the two meet in shared memory,
// and the first half of the threads evaluates the fluxes.
constexpr int kThreads = 2 * kEdgeBlock;
constexpr int kFaceBlock = 64;

// W = (Sigma, l, Pi) of the conserved state and the candidates of its dt
// (once after the state is set; afterwards the stage-2 update does both).
__global__ void __launch_bounds__(kFaceBlock) prepare_kernel(DevGeom G, DevState S, PhysParams P) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  double vel2 = 0.0, rate2 = 0.0;
  bool negative = false;
  if (f < G.n_faces) {
    double u[kDim], w[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) u[k] = S.U[k * G.fpad + f];
    const D3 r = plane3(G.fcn, G.fpad, f);
    prim_of(u, r, P.gam, w);
#pragma unroll
    for (int k = 0; k < kDim; ++k) S.W0[k * G.fpad + f] = w[k];
    dt_fold(w, r, P, vel2, rate2, negative);
  }
  fold_warp(vel2, rate2, negative, S, P, gridDim.x * (kFaceBlock / 32));
}

// the flux of edge e, whose sides are columns i and kEdgeBlock + i
__device__ __forceinline__ void store_flux(const DevGeom& G, const DevState& S, const PhysParams& P, const Gas& gas,
                                           const SideExchange<double, kThreads>& sides, int e, int i) {
  double L[kDim], R[kDim], F[kDim];
  EdgeSide<double> SL, SR;
  sides.get(i, L, SL);
  sides.get(kEdgeBlock + i, R, SR);
  unsigned bits = riemann_flux(L, R, SL, SR, edge_geom(G, e), gas, P.solver, F);
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    if (nan_bits(F[k])) bits |= 1u;
    S.fe[(size_t)k * G.epad + e] = F[k];
  }
  if (bits) atomicOr(S.err, bits);
}

// find_U_edges (MUSCL_base.hpp:361-434) of both sides of every edge and the
// Riemann flux (find_flux_var, MUSCL_base.hpp:345-359).
template <int STAGE>
__global__ void __launch_bounds__(kThreads) edge_kernel(DevGeom G, DevState S, PhysParams P, double dt0) {
  griddep_launch_dependents();
  __shared__ SideExchange<double, kThreads> sides;
  const int t = threadIdx.x, i = t & (kEdgeBlock - 1);
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const Gas gas = gas_of(P);
  if (live) {
    const int x = (t < kEdgeBlock) ? e : G.epad + e;
    const SideGeom g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[G.xs + x], G.e_sten[2 * G.xs + x], G.e_sten[3 * G.xs + x]};
    griddep_wait();
    const double dt = (STAGE == 1) ? step_dt(S.scal, dt0) : S.scal[kScDt];
    const double* W = (STAGE == 1) ? S.W0 : S.W1;
    const int fp = G.fpad;
    double w[kDim], u[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) w[k] = W[k * fp + f];
    recon_side(g, P.gam, dt, w, [&](int k, int q) { return W[k * fp + st[q]]; }, u);
    if (STAGE == 2) {
#pragma unroll
      for (int k = 0; k < kDim; ++k) S.uplus[(size_t)k * G.xs + x] = u[k];
    }
    if (STAGE == 1 && x == 0) publish_dt(S, dt);
    sides.put(t, u, edge_side(u, edge_geom(G, e), gas));
  }
  __syncthreads();
  if (!live || t >= kEdgeBlock) return;
  store_flux(G, S, P, gas, sides, e, i);
}

// The same with kDim threads per side, one per field, for meshes whose sides
// leave the SMs a warp or two: there a launch takes the latency of one
// thread's chain, 255 dependent FP64 instructions of 33 ns and 3,100 in all.
// Warp 2 k + s of a block serves field k of side s of its 32 edges; the field
// 0 warps evaluate the side's Courant factor while the others form their
// differences, then every warp limits its field, and the field 0 warps go on
// as in edge_kernel.  Two blocks per SM: at one (112 registers) hex(4) takes
// two waves, 51.6 us per step instead of 40.7.
template <int STAGE>
__global__ void __launch_bounds__(kEdgePartThreads, 2) edge_parts_kernel(DevGeom G, DevState S, PhysParams P, double dt0) {
  griddep_launch_dependents();
  __shared__ SideExchange<double, kThreads> sides;
  __shared__ double up[kDim][kThreads];
  __shared__ __align__(8) unsigned char limiters[kThreads * sizeof(SideLimiter)];
  const int warp = threadIdx.x / 32, k = warp >> 1, i = threadIdx.x & 31;
  const int t = (warp & 1) * kEdgeBlock + i;  // the side, as in edge_kernel
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const int x = (t < kEdgeBlock) ? e : G.epad + e;
  const size_t fp = G.fpad, xs = G.xs;
  SideLimiter& limiter = reinterpret_cast<SideLimiter*>(limiters)[t];
  SideGeom g{};
  double wk = 0.0, dp = 0.0, num = 0.0, dpg = 0.0;
  if (live) {
    g = side_geom(G, x);
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    griddep_wait();
    const double* W = (STAGE == 1) ? S.W0 : S.W1;
    const double* Wk = W + k * fp;
    wk = Wk[f];
    double dm;
    side_differences(g, wk, Wk[st[0]], Wk[st[1]], Wk[st[2]], Wk[st[3]], dp, dm);
    num = dm * g.hr;
    dpg = dp * g.hg;
    if (k == 0) {
      const double dt = (STAGE == 1) ? step_dt(S.scal, dt0) : S.scal[kScDt];
      double w[kDim], c;
#pragma unroll
      for (int q = 0; q < kDim; ++q) w[q] = W[q * fp + f];
      const double nu = side_courant(g, P.gam, dt, w, c);
      limiter = SideLimiter(g, nu, w[0], w[4], c);
    } else if (STAGE == 1 && k == kDim - 1 && x == 0) {
      publish_dt(S, step_dt(S.scal, dt0));
    }
  }
  __syncthreads();
  if (live) {
    double lim;
    if (!limiter.in_pairs(k, dp, num, dpg, lim)) {
      const LimiterLine<double> line = limiter_line(g.eta_p, g.sbs, limiter.nu);
      lim = limiter_full(dp, num, line.eta_p, line.sb, line.ts, line.t1);
    }
    const double u = fm(dpg, lim, wk);
    up[k][t] = u;
    if (STAGE == 2) S.uplus[k * xs + x] = u;
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
  store_flux(G, S, P, gas, sides, e, i);
}

// res2d + the RK combine; stage 1: dt/2, writes W1; stage 2: dt, writes U, W0
// and folds the candidates of the next dt.  This is the part after the sums
// and the source, of one face per lane; every lane of the warp calls it.
template <int STAGE>
__device__ __forceinline__ void finish_face(const DevGeom& G, const DevState& S, const PhysParams& P, int f, bool live,
                                            const double* src, const double* sum, unsigned long long n_warps) {
  double vel2 = 0.0, rate2 = 0.0;
  bool negative = false;
  if (live) {
    const int fp = G.fpad;
    const double dt = S.scal[kScDt];
    double u0[kDim], u[kDim], w[kDim];
#pragma unroll
    for (int k = 0; k < kDim; ++k) u0[k] = S.U[k * fp + f];
    bool floored;
    combine_face((STAGE == 1) ? 0.5 * dt : dt, src, sum, u0, u, floored);
    const D3 fcn = plane3(G.fcn, fp, f);
    prim_of(u, fcn, P.gam, w);
    double* Wout = (STAGE == 1) ? S.W1 : S.W0;
#pragma unroll
    for (int k = 0; k < kDim; ++k) Wout[k * fp + f] = w[k];
    if (STAGE == 2) {
#pragma unroll
      for (int k = 0; k < kDim; ++k) S.U[k * fp + f] = u[k];
      dt_fold(w, fcn, P, vel2, rate2, negative);
    }
  }
  if (STAGE == 2) fold_warp(vel2, rate2, negative, S, P, n_warps);
}
template <int STAGE>
__device__ __forceinline__ void face_source(const DevGeom& G, const DevState& S, const PhysParams& P, int f,
                                            double* src) {
  const double* Win = (STAGE == 1) ? S.W0 : S.W1;
  double w[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) w[k] = Win[k * G.fpad + f];
  source_term(w, plane3(G.fcn, G.fpad, f), face_src_params<double>(G, P, f), P, src);
}

// one thread per face
template <int STAGE>
__global__ void __launch_bounds__(kFaceBlock) update_kernel(DevGeom G, DevState S, PhysParams P) {
  griddep_launch_dependents();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = f < G.n_faces;
  double src[kDim] = {0, 0, 0, 0, 0}, sum[kDim] = {0, 0, 0, 0, 0};
  griddep_wait();
  if (live) {
    face_source<STAGE>(G, S, P, f, src);
    // flux_sum of the five fields in one walk over the slots
    const int n = G.nslots[f];
    for (int j = 0; j < n; ++j) {
      const int se = G.slot_edge[j * G.fpad + f];
      const int e = se & 0x7fffffff;
      const double c = G.e_side[(size_t)kSideCoef * G.xs + (se < 0 ? G.epad + e : e)];
#pragma unroll
      for (int k = 0; k < kDim; ++k) sum[k] = fma((se < 0) ? c : -c, S.fe[(size_t)k * G.epad + e], sum[k]);
    }
  }
  finish_face<STAGE>(G, S, P, f, live, src, sum, gridDim.x * (kFaceBlock / 32));
}
// kDim + 1 threads per face (face_part)
template <int STAGE, int BLOCKS>
__global__ void __launch_bounds__(kFaceThreads, BLOCKS) update_parts_kernel(DevGeom G, DevState S, PhysParams P) {
  griddep_launch_dependents();
  __shared__ FaceParts<double, 2 * kDim> parts;
  const int part = face_part(), i = threadIdx.x % kFaces, f = blockIdx.x * kFaces + i;
  const bool live = f < G.n_faces;
  FluxTerms terms;
  if (live && part < kDim) terms = flux_terms(G, f);
  griddep_wait();
  if (live && part < kDim) {
    const double* fe = S.fe + (size_t)part * G.epad;
    parts.put(part, i, flux_sum<double>(G, f, terms, [&](int e) { return fe[e]; }));
  } else if (live) {
    double src[kDim];
    face_source<STAGE>(G, S, P, f, src);
#pragma unroll
    for (int k = 0; k < kDim; ++k) parts.put(kDim + k, i, src[k]);
  }
  __syncthreads();
  if (part != 0) return;
  double src[kDim], sum[kDim];
#pragma unroll
  for (int k = 0; k < kDim; ++k) {
    sum[k] = live ? parts.get(k, i) : 0.0;
    src[k] = live ? parts.get(kDim + k, i) : 0.0;
  }
  finish_face<STAGE>(G, S, P, f, live, src, sum, gridDim.x);
}

// ---- isothermal solver (MUSCL_HLLE, 4 fields; planes 0..3 of U/W/U+) ----
// W of a 4-field state is the state itself (find_U_edges subtracts the
// zero profile rho_an from field 0, MUSCL_base.hpp:366-371).
__global__ void __launch_bounds__(kFaceBlock) iso_prepare_kernel(DevGeom G, DevState S, PhysParams P) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  double vel2 = 0.0;
  if (f < G.n_faces) {
    double u[iso::kIsoDim];
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) {
      u[k] = S.U[k * G.fpad + f];
      S.W0[k * G.fpad + f] = u[k];
    }
    vel2 = iso::dt_fold(u, plane3(G.fcn, G.fpad, f));
  }
  fold_warp(vel2, 0.0, false, S, P, gridDim.x * (kFaceBlock / 32));
}

// the two sides' states with the isothermal limiter (MUSCL_base.hpp:361-434,
// physics/isothermal.hpp:269-320) and the HLLE flux of every edge
template <int STAGE>
__global__ void __launch_bounds__(kThreads) iso_edge_kernel(DevGeom G, DevState S, PhysParams P, double dt0) {
  griddep_launch_dependents();
  __shared__ double up[iso::kIsoDim][kThreads];
  const int t = threadIdx.x, i = t & (kEdgeBlock - 1);
  const int e = blockIdx.x * kEdgeBlock + i;
  const bool live = e < G.n_edges;
  const size_t ep = (size_t)G.epad, xs = (size_t)G.xs;
  const D3 ec = live ? D3{G.e_geo[e], G.e_geo[ep + e], G.e_geo[2 * ep + e]} : D3{0, 0, 0};
  if (live) {
    const int x = (t < kEdgeBlock) ? e : G.epad + e;
    const double* c = G.e_side + x;
    const int f = G.e_face[x];
    const int st[4] = {G.e_sten[x], G.e_sten[xs + x], G.e_sten[2 * xs + x], G.e_sten[3 * xs + x]};
    const double twoN = (double)(2 * G.nslots[f]);
    griddep_wait();
    const double dt = (STAGE == 1) ? step_dt(S.scal, dt0) : S.scal[kScDt];
    const double* W = (STAGE == 1) ? S.W0 : S.W1;
    const int fp = G.fpad;
    double w[iso::kIsoDim];
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) w[k] = W[k * fp + f];
    const D3 en = D3{c[kIsoEn * xs], c[(kIsoEn + 1) * xs], c[(kIsoEn + 2) * xs]};
    const iso::Limiter lim(c[kIsoEta * xs], twoN, iso::courant(w, ec, en, dt, c[kIsoArc * xs]));
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) {
      const double* Wk = W + k * fp;
      const double Up = c[kSideBeta * xs] * Wk[st[0]] + c[(kSideBeta + 1) * xs] * Wk[st[1]];
      const double pp = quotient(Up - w[k], c[kIsoHp * xs], c[kIsoRhp * xs]);
      const double Um = c[(kSideBeta + 2) * xs] * Wk[st[2]] + c[(kSideBeta + 3) * xs] * Wk[st[3]];
      const double pm = quotient(-Um + w[k], c[kIsoHm * xs], c[kIsoRhm * xs]);
      const double u = w[k] + pp * lim(divide(pm, pp)) * c[kIsoBm * xs];
      up[k][t] = u;
      if (STAGE == 2) S.uplus[k * xs + x] = u;
    }
    if (STAGE == 1 && x == 0) publish_dt(S, dt);
  }
  __syncthreads();
  if (!live || t >= kEdgeBlock) return;
  double L[iso::kIsoDim], R[iso::kIsoDim], F[iso::kIsoDim];
#pragma unroll
  for (int k = 0; k < iso::kIsoDim; ++k) {
    L[k] = up[k][i];
    R[k] = up[k][kEdgeBlock + i];
  }
  unsigned bits = iso::flux_star(L, R, ec, G.e_geo[6 * ep + e],
                                 D3{G.e_geo[3 * ep + e], G.e_geo[4 * ep + e], G.e_geo[5 * ep + e]}, F);
#pragma unroll
  for (int k = 0; k < iso::kIsoDim; ++k) {
    if (nan_bits(F[k])) bits |= 1u;
    S.fe[k * ep + e] = F[k];
  }
  if (bits) atomicOr(S.err, bits);
}

// res2d + the RK combine (zero source) for one face
template <int STAGE>
__global__ void __launch_bounds__(kFaceBlock) iso_update_kernel(DevGeom G, DevState S, PhysParams P) {
  griddep_launch_dependents();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  double vel2 = 0.0;
  griddep_wait();
  if (f < G.n_faces) {
    const int fp = G.fpad;
    const double dt = S.scal[kScDt];
    const double dt_here = (STAGE == 1) ? dt / 2 : dt;
    const double area = G.area[f], iarea = recip(area);
    double u[iso::kIsoDim];
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) u[k] = 0.0;
    const double rd_dt = P.round_diff * dt_here;
    const int n = G.nslots[f];
    for (int j = 0; j < n; ++j) {
      const int se = G.slot_edge[j * fp + f];
      const int e = se & 0x7fffffff;
      const double chord = G.e_side[(size_t)kIsoChord * G.xs + (se < 0 ? G.epad + e : e)];
      const double q = quotient(rd_dt * chord, area, iarea);
      const double coef = (se < 0) ? -q : q;
#pragma unroll
      for (int k = 0; k < iso::kIsoDim; ++k) u[k] -= coef * S.fe[(size_t)k * G.epad + e];
    }
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) u[k] = u[k] + S.U[k * fp + f];
    if (u[0] < 1e-8) u[0] = 1e-8;
    double* Wout = (STAGE == 1) ? S.W1 : S.W0;
#pragma unroll
    for (int k = 0; k < iso::kIsoDim; ++k) {
      Wout[k * fp + f] = u[k];
      if (STAGE == 2) S.U[k * fp + f] = u[k];
    }
    if (STAGE == 2) vel2 = iso::dt_fold(u, plane3(G.fcn, fp, f));
  }
  if (STAGE == 2) fold_warp(vel2, 0.0, false, S, P, gridDim.x * (kFaceBlock / 32));
}

// reference order [F][dim] <-> internal planes
// One thread per element of the [n_faces][dim] array, in its memory order,
// so that every warp reads or writes 256 contiguous bytes of it -- device
// memory or, on a coherent host link, the caller's host memory, where
// partial-line accesses are expensive; the planes take the permuted side.
// (dim = 4: the fifth plane is written as zero by the scatter.)
__global__ void scatter_state_kernel(const double* __restrict__ aos, const int* __restrict__ iperm,
                                     double* __restrict__ U, int n_faces, int fpad, int dim) {
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= (size_t)n_faces * dim) return;
  const int r = (int)(e / dim), k = (int)(e % dim);
  const int i = iperm[r];
  U[(size_t)k * fpad + i] = aos[e];
  if (dim == 4 && k == 3) U[(size_t)4 * fpad + i] = 0.0;
}
__global__ void gather_state_kernel(const double* __restrict__ U, const int* __restrict__ iperm,
                                    double* __restrict__ aos, int n_faces, int fpad, int dim) {
  const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (e >= (size_t)n_faces * dim) return;
  const int r = (int)(e / dim), k = (int)(e % dim);
  aos[e] = U[(size_t)k * fpad + iperm[r]];
}
// Two consecutive elements per thread with one 16-byte access on the
// caller's side (used when the caller's array is 16-byte aligned): half the
// warp instructions on the host link, 512 contiguous bytes per warp access.
__global__ void gather_state2_kernel(const double* __restrict__ U, const int* __restrict__ iperm,
                                     double* __restrict__ aos, int n_faces, int fpad, int dim) {
  const unsigned ne = (unsigned)n_faces * (unsigned)dim;
  const unsigned e0 = 2u * (blockIdx.x * blockDim.x + threadIdx.x);
  if (e0 >= ne) return;
  double v[2] = {0.0, 0.0};
#pragma unroll
  for (unsigned q = 0; q < 2; ++q) {
    const unsigned e = e0 + q;
    if (e < ne) {
      const unsigned r = e / (unsigned)dim, k = e - r * (unsigned)dim;
      v[q] = U[(size_t)k * fpad + iperm[r]];
    }
  }
  if (e0 + 1 < ne)
    *reinterpret_cast<double2*>(aos + e0) = make_double2(v[0], v[1]);
  else
    aos[e0] = v[0];
}
constexpr int kMoveBlock = 256;

inline int face_blocks(int n, int per = kFaceBlock) { return (n + per - 1) / per; }
inline int edge_blocks(int n) { return (n + kEdgeBlock - 1) / kEdgeBlock; }

}  // namespace
}  // namespace f64

// ---- launchers (declared in kernels.hpp) --------------------------------
cudaError_t fp64_prepare(const DevGeom& G, const DevState& S, const PhysParams& P, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(S.fold, 0, kFoldCount * sizeof(*S.fold), st);
  if (e != cudaSuccess) return e;
  if (P.solver == kSolverIsoHLLE)
    f64::iso_prepare_kernel<<<f64::face_blocks(G.n_faces), f64::kFaceBlock, 0, st>>>(G, S, P);
  else
    f64::prepare_kernel<<<f64::face_blocks(G.n_faces), f64::kFaceBlock, 0, st>>>(G, S, P);
  return cudaGetLastError();
}

namespace {
// kDim threads per side on meshes of at most a wave and a quarter of its
// blocks (two per SM).  us per step of MUSCL_HLLE_p / HLLC+, one thread per
// side / kDim: hex(3) 48.8 / 37.5 and 54.5 / 43.3, hex(4) 53.9 / 40.7 and 59.7
// / 45.8, quad(5) (12,288 edges) 58.8 / 55.0 and 67.2 / 66.1; hex(5) (30,720)
// 72.3 / 122 and 81.6 / 160.
constexpr int kEdgePartsEdges = 12288;
bool edge_parts(const DevGeom& G) { return G.n_edges <= kEdgePartsEdges; }
}  // namespace

const void* fp64_dt0_kernel_ptr(const DevGeom& G, int solver) {
  return solver == kSolverIsoHLLE ? (const void*)f64::iso_edge_kernel<1>
         : edge_parts(G)          ? (const void*)f64::edge_parts_kernel<1>
                                  : (const void*)f64::edge_kernel<1>;
}

cudaError_t fp64_step(const DevGeom& G, const DevState& S, const PhysParams& P, double dt0, cudaStream_t st,
                      cudaEvent_t* ev) {
  using Edge = void (*)(DevGeom, DevState, PhysParams, double);
  using Update = void (*)(DevGeom, DevState, PhysParams);
  // six threads per face where one per face leaves the pipe to a warp or two
  // per SM; where it does not, the combining warp's share of a block's
  // registers costs more.  us per step, one / six: hex(4) 53.9 / 52.4, hex(5)
  // 97 / 76 (shear 131 / 97), hex(6) (40,962 faces) 250 / 224, quad(7) (98,304)
  // 366 / 367, hex(7) 760 / 798, quad(8) 1262 / 1352.
  constexpr int kPartsFaces = 65536;
  const bool iso = P.solver == kSolverIsoHLLE, parts = !iso && G.n_faces <= kPartsFaces;
  const bool fields = !iso && edge_parts(G);
  const Edge edge1 = iso ? f64::iso_edge_kernel<1> : fields ? f64::edge_parts_kernel<1> : f64::edge_kernel<1>;
  const Edge edge2 = iso ? f64::iso_edge_kernel<2> : fields ? f64::edge_parts_kernel<2> : f64::edge_kernel<2>;
  const bool five = parts && f64::five_face_blocks(G.n_faces);
  const Update upd1 = iso     ? f64::iso_update_kernel<1>
                      : five  ? f64::update_parts_kernel<1, 5>
                      : parts ? f64::update_parts_kernel<1, 4>
                              : f64::update_kernel<1>;
  const Update upd2 = iso     ? f64::iso_update_kernel<2>
                      : five  ? f64::update_parts_kernel<2, 5>
                      : parts ? f64::update_parts_kernel<2, 4>
                              : f64::update_kernel<2>;
  const dim3 eg(f64::edge_blocks(G.n_edges)), eb(fields ? f64::kEdgePartThreads : f64::kThreads);
  const dim3 fg(f64::face_blocks(G.n_faces, parts ? f64::kFaces : f64::kFaceBlock));
  const dim3 fb(parts ? f64::kFaceThreads : f64::kFaceBlock);
  FirstError chk;
  // ev[0]..ev[1] is the (empty) slot of the dt clip, which the stage-1 edge
  // launch evaluates itself
  if (ev) cudaEventRecord(ev[0], st);
  if (ev) cudaEventRecord(ev[1], st);
  chk(launch_pdl(edge1, eg, eb, st, G, S, P, dt0));
  if (ev) cudaEventRecord(ev[2], st);
  chk(launch_pdl(upd1, fg, fb, st, G, S, P));
  if (ev) cudaEventRecord(ev[3], st);
  chk(launch_pdl(edge2, eg, eb, st, G, S, P, dt0));
  if (ev) cudaEventRecord(ev[4], st);
  chk(launch_pdl(upd2, fg, fb, st, G, S, P));
  if (ev) cudaEventRecord(ev[5], st);
  return chk.status();
}

cudaError_t fp64_scatter_state(const double* aos, const int* iperm, double* U, int n_faces,
                               int fpad, cudaStream_t st, int dim) {
  const size_t ne = (size_t)n_faces * dim;
  f64::scatter_state_kernel<<<(unsigned)((ne + f64::kMoveBlock - 1) / f64::kMoveBlock), f64::kMoveBlock, 0, st>>>(
      aos, iperm, U, n_faces, fpad, dim);
  return cudaGetLastError();
}

cudaError_t fp64_gather_state(const double* U, const int* iperm, double* aos, int n_faces,
                              int fpad, cudaStream_t st, int dim) {
  const size_t ne = (size_t)n_faces * dim;
  if (((uintptr_t)aos & 15) == 0) {
    const size_t nt = (ne + 1) / 2;
    f64::gather_state2_kernel<<<(unsigned)((nt + f64::kMoveBlock - 1) / f64::kMoveBlock), f64::kMoveBlock, 0, st>>>(
        U, iperm, aos, n_faces, fpad, dim);
    return cudaGetLastError();
  }
  f64::gather_state_kernel<<<(unsigned)((ne + f64::kMoveBlock - 1) / f64::kMoveBlock), f64::kMoveBlock, 0, st>>>(
      U, iperm, aos, n_faces, fpad, dim);
  return cudaGetLastError();
}

}  // namespace splash
