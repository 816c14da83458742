// Host preparation of the device layout; see slot_planes.hpp.
#include "slot_planes.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>

#include "hilbert.hpp"
#include "layout.hpp"

namespace splash {

namespace {
struct V3 {
  double x, y, z;
};
inline V3 vadd(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
inline V3 vsub(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
inline V3 vdiv(V3 a, double s) { return {a.x / s, a.y / s, a.z / s}; }
inline double vnorm(V3 a) {
  double s = 0.0;
  s += a.x * a.x;
  s += a.y * a.y;
  s += a.z * a.z;
  return std::sqrt(s);
}
inline V3 vcross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
inline V3 at3(const std::vector<double>& v, size_t i) { return {v[3 * i], v[3 * i + 1], v[3 * i + 2]}; }
}  // namespace

SlotPlanes make_slot_planes(const RefGeometry& g) {
  SlotPlanes sp;
  const int nf = g.n_faces;
  const int max_slots = g.max_slots;
  const int fpad = (nf + 31) / 32 * 32;
  sp.n_faces = nf;
  sp.max_slots = max_slots;
  sp.fpad = fpad;
  sp.round_diff = g.round_diff;
  const size_t PS = sp.PS();

  sp.perm = hilbert_order(g.face_centers.data(), nf);
  sp.iperm.assign(nf, 0);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < nf; ++i) sp.iperm[sp.perm[i]] = i;
  const std::vector<int>& perm = sp.perm;
  const std::vector<int>& iperm = sp.iperm;

  // reference-order reverse slot (std::find of MUSCL_base.hpp:383-384)
  std::vector<int> j0_of(g.n_slots, -1);
  bool asymmetric = false;
#pragma omp parallel for schedule(static) reduction(|| : asymmetric)
  for (int f = 0; f < nf; ++f) {
    for (int s = g.face_off[f]; s < g.face_off[f + 1]; ++s) {
      const int nb = g.nbr_edge[s];
      int j0 = -1;
      for (int q = g.face_off[nb]; q < g.face_off[nb + 1]; ++q)
        if (g.nbr_edge[q] == f) {
          j0 = q - g.face_off[nb];
          break;
        }
      if (j0 < 0) asymmetric = true;
      j0_of[s] = j0;
    }
  }
  if (asymmetric) throw std::runtime_error("edge neighbour relation is not symmetric");

  sp.nslots.assign(fpad, 0);
  sp.fcn.assign(3 * (size_t)fpad, 0.0);
  sp.area.assign(fpad, 1.0);
  sp.sten.resize(4 * PS);
  sp.rev.resize(PS);
  sp.beta.resize(4 * PS);
  sp.hpm.resize(2 * PS);
  sp.bm.resize(PS);
  sp.eta.resize(2 * PS);
  sp.arc.resize(PS);
  sp.ec.resize(3 * PS);
  sp.ecn.resize(PS);
  sp.en.resize(3 * PS);
  sp.nxr.resize(3 * PS);
  sp.chord.resize(PS);

  // every face writes only its own entries: the fill is order-independent
#pragma omp parallel for schedule(static)
  for (int i = 0; i < nf; ++i) {
    const int r = perm[i];
    const int n = g.face_off[r + 1] - g.face_off[r];
    sp.nslots[i] = (int8_t)n;
    const V3 fc = at3(g.face_centers, r);
    const V3 fcn = vdiv(fc, vnorm(fc));
    sp.fcn[i] = fcn.x;
    sp.fcn[fpad + i] = fcn.y;
    sp.fcn[2 * (size_t)fpad + i] = fcn.z;
    sp.area[i] = g.area[r];
    for (int j = 0; j < n; ++j) {
      const int sr = g.face_off[r] + j;
      const size_t s = (size_t)j * fpad + i;
      sp.sten[s] = iperm[g.ff_plus[2 * (size_t)sr]];
      sp.sten[PS + s] = iperm[g.ff_plus[2 * (size_t)sr + 1]];
      sp.sten[2 * PS + s] = iperm[g.ff_minus[2 * (size_t)sr]];
      sp.sten[3 * PS + s] = iperm[g.ff_minus[2 * (size_t)sr + 1]];
      sp.beta[s] = g.beta_plus[2 * (size_t)sr];
      sp.beta[PS + s] = g.beta_plus[2 * (size_t)sr + 1];
      sp.beta[2 * PS + s] = g.beta_minus[2 * (size_t)sr];
      sp.beta[3 * PS + s] = g.beta_minus[2 * (size_t)sr + 1];
      sp.hpm[s] = g.h_plus[sr];
      sp.hpm[PS + s] = g.h_minus[sr];
      sp.bm[s] = g.bm_dist[sr];
      sp.eta[s] = g.h_plus[sr] / g.bm_dist[sr];
      sp.eta[PS + s] = g.h_minus[sr] / g.bm_dist[sr];
      const int va = g.face_vtx[sr];
      const int vb = g.face_vtx[g.face_off[r] + ((j + 1 == n) ? 0 : j + 1)];
      const V3 A = at3(g.vertices, va), B = at3(g.vertices, vb);
      // great-circle edge length / area: the limiter's Courant factor
      // (physics/adiabatic.hpp:757-758)
      sp.arc[s] = great_circle(&g.vertices[3 * (size_t)va], &g.vertices[3 * (size_t)vb]) / g.area[r];
      V3 ec = vdiv(vadd(A, B), 2.);
      ec = vdiv(ec, vnorm(ec));
      const double ecn = vnorm(ec);
      sp.ec[s] = ec.x;
      sp.ec[PS + s] = ec.y;
      sp.ec[2 * PS + s] = ec.z;
      sp.ecn[s] = ecn;
      const V3 en = at3(g.edge_normals, sr);
      sp.en[s] = en.x;
      sp.en[PS + s] = en.y;
      sp.en[2 * PS + s] = en.z;
      const V3 nxr = vcross(en, vdiv(ec, ecn));
      sp.nxr[s] = nxr.x;
      sp.nxr[PS + s] = nxr.y;
      sp.nxr[2 * PS + s] = nxr.z;
      sp.chord[s] = vnorm(vsub(A, B));
      sp.rev[s] = j0_of[sr] * fpad + iperm[g.nbr_edge[sr]];
    }
    // unused slots of low-valence faces point at themselves (never read)
    for (int j = n; j < max_slots; ++j) {
      const size_t s = (size_t)j * fpad + i;
      for (int q = 0; q < 4; ++q) sp.sten[q * PS + s] = i;
      sp.rev[s] = (int)s;
    }
  }
  return sp;
}

double area_coefficient(const RefGeometry& g, double acc_width) {
  double ac = 0;
  const double mu = M_PI / 2;
  const double sigma = acc_width / 2.355;
  for (int n = 0; n < g.n_faces; ++n) {
    const V3 c = at3(g.face_centers, n);
    const double theta = std::acos(c.z / vnorm(c));
    ac += g.area[n] / std::sqrt(2 * M_PI * sigma * sigma) *
          std::exp(-(theta - mu) * (theta - mu) / (2 * sigma * sigma));
  }
  ac /= 4 * M_PI;
  return ac;
}

std::vector<double> accretion_source(const SlotPlanes& sp, const splash_params& par,
                                     double area_coeff, bool accretion_on) {
  return accretion_source_fcn(sp.fcn, sp.n_faces, sp.fpad, par, area_coeff, accretion_on);
}

std::vector<double> accretion_source_fcn(const std::vector<double>& fcn, int n_faces, int fpad,
                                         const splash_params& par, double area_coeff, bool accretion_on,
                                         std::vector<double>* d_rate, std::vector<double>* d_tilt) {
  std::vector<double> acc(fpad, 0.0);
  if (d_rate) d_rate->assign(fpad, 0.0);
  if (d_tilt) d_tilt->assign(fpad, 0.0);
  if (!accretion_on) return acc;
  const double sigma = par.acc_width / 2.355;
  const double mu = M_PI / 2;
  const double st = std::sin(par.tilt_angle), ct = std::cos(par.tilt_angle);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n_faces; ++i) {
    const V3 c{fcn[i], fcn[fpad + i], fcn[2 * (size_t)fpad + i]};
    const double x = c.y * std::sin(par.tilt_angle) + c.z * std::cos(par.tilt_angle);
    const double theta_acc = std::acos(x);
    const double g = std::exp(-(theta_acc - mu) * (theta_acc - mu) / (2 * sigma * sigma));
    acc[i] = 1 / area_coeff * par.accretion_rate / std::sqrt(2 * M_PI * sigma * sigma) * g;
    // d acc / d rate, and d acc / d tilt through theta_acc = acos(x)
    if (d_rate) (*d_rate)[i] = 1 / area_coeff / std::sqrt(2 * M_PI * sigma * sigma) * g;
    if (d_tilt) {
      const double dx = c.y * ct - c.z * st;
      const double s2 = 1 - x * x;
      const double dtheta = (s2 > 0) ? -dx / std::sqrt(s2) : 0.0;
      (*d_tilt)[i] = acc[i] * (-(theta_acc - mu) / (sigma * sigma)) * dtheta;
    }
  }
  return acc;
}

EdgeList make_edge_list(const SlotPlanes& sp) {
  EdgeList el;
  const size_t PS = sp.PS();
  // Owner slots: of the two slots of an edge, the one with the smaller
  // slot-plane index.  Edge e is the e-th owner slot in the visiting order
  // below, its index an exclusive prefix sum of the owner flags.
  std::vector<unsigned char> is_own(PS, 0);
  bool lonely = false;
#pragma omp parallel for schedule(static) reduction(|| : lonely)
  for (long long q = 0; q < (long long)PS; ++q) {
    const int i = (int)(q % sp.fpad), j = (int)(q / sp.fpad);
    if (i >= sp.n_faces || j >= (int)sp.nslots[i]) continue;
    const int r = sp.rev[q];
    if (r == (int)q) lonely = true;
    is_own[q] = (int)q < r;
  }
  if (lonely) throw std::runtime_error("slot without a neighbour");
  // Edges numbered face-major: the owner face's internal (Hilbert) index,
  // then its slot, so that the edges of a run of faces form one compact
  // range (the update's flux gathers stay local; measured 1% faster per step
  // on hex(7) than ascending slot-plane order).  Prefix sum over fixed chunks
  // of faces: counts per chunk, then offsets.
  const long long nvisit = (long long)sp.n_faces;
  const int ms = sp.max_slots, fp = sp.fpad;
  auto visit = [&](long long v, auto&& fn) {  // the owner-candidate slots of face v, in slot order
    for (int j = 0; j < ms; ++j) fn((long long)j * fp + v);
  };
  const long long nchunk = 256, clen = (nvisit + nchunk - 1) / nchunk;
  std::vector<long long> base(nchunk + 1, 0);
#pragma omp parallel for schedule(static)
  for (long long c = 0; c < nchunk; ++c) {
    long long cnt = 0;
    for (long long v = c * clen; v < std::min(nvisit, (c + 1) * clen); ++v)
      visit(v, [&](long long q) { cnt += is_own[q]; });
    base[c + 1] = cnt;
  }
  for (long long c = 0; c < nchunk; ++c) base[c + 1] += base[c];
  el.n_edges = (int)base[nchunk];
  el.own.resize(el.n_edges);
  el.nbr.resize(el.n_edges);
  el.slot_edge.assign(PS, 0);
#pragma omp parallel for schedule(static)
  for (long long c = 0; c < nchunk; ++c) {
    long long e = base[c];
    for (long long v = c * clen; v < std::min(nvisit, (c + 1) * clen); ++v)
      visit(v, [&](long long q) {
        if (!is_own[q]) return;
        const int r = sp.rev[q];
        el.own[e] = (int)q;
        el.nbr[e] = r;
        el.slot_edge[q] = (int)e;
        el.slot_edge[r] = (int)((unsigned)e | 0x80000000u);
        ++e;
      });
  }
  return el;
}

int padded_edges(int n_edges) {
  const size_t pad = ((size_t)n_edges + kEdgeBlock - 1) / kEdgeBlock * kEdgeBlock;
  if (2 * pad > kMaxSides) throw std::runtime_error("too many edges");
  return (int)pad;
}

EdgePlanes make_edge_planes(const SlotPlanes& sp, bool isothermal) {
  EdgePlanes ep;
  const size_t PS = sp.PS();
  bool paired = true;
#pragma omp parallel for schedule(static) reduction(&& : paired)
  for (int i = 0; i < sp.n_faces; ++i)
    for (int j = 0; j < (int)sp.nslots[i]; ++j) {
      const size_t q = (size_t)j * sp.fpad + i, r = (size_t)sp.rev[q];
      bool ok = r != q && (size_t)sp.rev[r] == q;
      for (size_t c = 0; c < 3; ++c)
        ok = ok && sp.en[c * PS + q] == -sp.en[c * PS + r] && sp.ec[c * PS + q] == sp.ec[c * PS + r];
      paired = paired && ok;
    }
  EdgeList el;
  if (paired) {
    el = make_edge_list(sp);
  } else {
    el.slot_edge.assign(PS, 0);
    for (int i = 0; i < sp.n_faces; ++i)
      for (int j = 0; j < (int)sp.nslots[i]; ++j) {
        const size_t q = (size_t)j * sp.fpad + i;
        el.slot_edge[q] = (int)el.own.size();
        el.own.push_back((int)q);
        el.nbr.push_back(sp.rev[q]);
      }
    el.n_edges = (int)el.own.size();
    for (int q : el.nbr) ep.twin.push_back(el.slot_edge[q]);
  }
  const int ne = ep.n_edges = el.n_edges;
  const size_t pad = ep.epad = padded_edges(ne), xs = 2 * pad;
  ep.slot_edge = std::move(el.slot_edge);
  ep.face.resize(xs);
  ep.sten.resize(4 * xs);
  ep.side.resize((size_t)(isothermal ? kIsoPlanes : kSidePlanes) * xs);
  ep.geo.resize(7 * pad);
#pragma omp parallel for schedule(static)
  for (int e = 0; e < ne; ++e) {
    const size_t so = (size_t)el.own[e];
    for (size_t c = 0; c < 3; ++c) {
      ep.geo[c * pad + e] = sp.ec[c * PS + so];
      ep.geo[(3 + c) * pad + e] = sp.en[c * PS + so];
    }
    ep.geo[6 * pad + e] = sp.ecn[so];
    for (int k = 0; k < 2; ++k) {
      const size_t q = k ? (size_t)el.nbr[e] : so, x = k * pad + e;
      const int f = (int)(q % sp.fpad);
      double* s = &ep.side[x];
      auto put = [&](int plane, double v) { s[(size_t)plane * xs] = v; };
      ep.face[x] = f;
      for (size_t c = 0; c < 4; ++c) {
        ep.sten[c * xs + x] = sp.sten[c * PS + q];
        put(kSideBeta + (int)c, sp.beta[c * PS + q]);
      }
      const double hp = sp.hpm[q], hm = sp.hpm[PS + q];
      if (isothermal) {
        put(kIsoHp, hp);
        put(kIsoHm, hm);
        put(kIsoRhp, 1.0 / hp);
        put(kIsoRhm, 1.0 / hm);
        put(kIsoArc, sp.arc[q]);
        for (int c = 0; c < 3; ++c) put(kIsoEn + c, sp.en[c * PS + q]);
        put(kIsoChord, sp.chord[q]);
        put(kIsoBm, sp.bm[q]);
        put(kIsoEta, sp.eta[PS + q]);
        continue;
      }
      put(kSideHr, hp / hm);
      put(kSideHg, sp.bm[q] / hp);
      put(kSideEtaP, sp.eta[q]);
      put(kSideSbs, sp.eta[PS + q] / (2 * sp.nslots[f]));
      put(kSideArc, sp.arc[q]);
      for (int c = 0; c < 3; ++c) put(kSideNxr + c, sp.nxr[c * PS + q]);
      // round_diff * chord / area with one rounding (the product's error and
      // the quotient's remainder put back)
      const double a = sp.area[f], p = sp.round_diff * sp.chord[q], c0 = p / a;
      const double coef = c0 + (std::fma(-c0, a, p) + std::fma(sp.round_diff, sp.chord[q], -p)) / a;
      put(kSideCoef, (k == 0 || paired) ? coef : 0.0);
    }
  }
  return ep;
}

MixedPlanes make_mixed_planes(const SlotPlanes& sp) {
  MixedPlanes mp;
  const size_t PS = sp.PS();
  mp.fcn32.assign(sp.fcn.begin(), sp.fcn.end());
  mp.fcn_lo.resize(sp.fcn.size());
  for (size_t i = 0; i < sp.fcn.size(); ++i) mp.fcn_lo[i] = (float)(sp.fcn[i] - (double)mp.fcn32[i]);
  mp.coef.assign(PS, 0.0f);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < sp.n_faces; ++i)
    for (int j = 0; j < (int)sp.nslots[i]; ++j) {
      const size_t q = (size_t)j * sp.fpad + i;
      mp.coef[q] = (float)(sp.round_diff * sp.chord[q] / sp.area[i]);
    }
  if (sp.n_faces >= (1 << 28)) throw std::runtime_error("too many faces for the edge records");
  const EdgeList el = make_edge_list(sp);
  const std::vector<int>&own = el.own, &nbr = el.nbr;
  mp.n_edges = el.n_edges;
  mp.slot_edge = el.slot_edge;
  const int ep = mp.epad = (mp.n_edges + 31) / 32 * 32;
  mp.e_ids.assign(4 * (size_t)ep, 0);
  mp.e_ec.assign(4 * (size_t)ep, 0.f);
  mp.e_en.assign(4 * (size_t)ep, 0.f);
  mp.e_sten.assign(8 * (size_t)ep, 0);
  mp.e_beta.assign(8 * (size_t)ep, 0.f);
  mp.e_h.assign(8 * (size_t)ep, 0.f);
#pragma omp parallel for schedule(static)
  for (int e = 0; e < mp.n_edges; ++e) {
    const size_t side_slot[2] = {(size_t)own[e], (size_t)nbr[e]};
    int face[2], n[2];
    for (int k = 0; k < 2; ++k) {
      face[k] = (int)(side_slot[k] % sp.fpad);
      n[k] = sp.nslots[face[k]];
    }
    int* id = &mp.e_ids[4 * (size_t)e];
    id[0] = face[0] | (n[0] << 28);
    id[1] = face[1] | (n[1] << 28);
    const size_t so = side_slot[0];
    for (int c = 0; c < 3; ++c) {
      mp.e_ec[4 * (size_t)e + c] = (float)sp.ec[c * PS + so];
      mp.e_en[4 * (size_t)e + c] = (float)sp.en[c * PS + so];
    }
    // the owner's n x R (FP64, rounded once) rides in the spare lanes
    mp.e_ec[4 * (size_t)e + 3] = (float)sp.nxr[so];
    mp.e_en[4 * (size_t)e + 3] = (float)sp.nxr[PS + so];
    const float nz = (float)sp.nxr[2 * PS + so];
    std::memcpy(&id[2], &nz, 4);
    id[3] = 0;
    for (int k = 0; k < 2; ++k) {
      const size_t q = side_slot[k];
      const size_t o = 4 * ((size_t)k * ep + e);
      for (int c = 0; c < 4; ++c) {
        mp.e_sten[o + c] = sp.sten[c * PS + q];
        mp.e_beta[o + c] = (float)sp.beta[c * PS + q];
      }
      mp.e_h[o + 0] = (float)(1.0 / sp.hpm[q]);
      mp.e_h[o + 1] = (float)(1.0 / sp.hpm[PS + q]);
      mp.e_h[o + 2] = (float)sp.bm[q];
      mp.e_h[o + 3] = (float)sp.arc[q];
    }
  }
  return mp;
}

}  // namespace splash
