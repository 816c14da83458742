// The limiter of the FP64 path in pairs of floats.
//
// The limited edge state is w + (dp BM / H+) lim, and lim, the limiter's value,
// meets the state only through the product with the difference dp.  Where that
// difference is below 2^-8 of the state, an error of 2^-45 in lim is 2^-53 of
// the state at most, the sum's own rounding.  There lim is evaluated in pairs
// of floats (an unevaluated sum of a float and its remainder, 48 bits), on the
// pipes that the FP64 work leaves idle: a product of pairs is 7 instructions
// of 1 cycle, an FP64 one 64 cycles (fp64_math.cuh).  The ratio r = (dm / H-)
// / (dp / H+) and its distance from 1 come from two FP64 differences, so that
// neither cancels.  Steeper differences, and ratios too far from the range of
// a float, take the FP64 evaluation (limiter_field).
//
// Per side of an edge 168 FP64 instructions instead of 252 (hex(7), HLLC+):
// edge launch 470 -> 315 us, step 1.05 -> 0.75 ms.  A bound of 2^-9 instead of
// 2^-8 leaves the error as it is and costs 8% where the flow is rough.  Over 4
// million ratios lim is within 2^-44.9 of an 80-bit evaluation (values up to
// 2.3).  The scale of l is Sigma c, not l: in slow flow a limited l is good to
// 2^-45 of its own difference, but the momentum flux carries Pi beside it.  The
// states bear that out: over 105 runs of 1 and 6 steps (4 flows, also at a
// thousandth of their speed, 3 solvers, hex and quad) their error against 80
// bits, over that of CUDA's operators and libm throughout, is 1.00 for Sigma
// and E and 0.93 for l.  The tangents of rough flows against a quad-precision
// difference quotient (36 runs): 0.91 by the median of the faces, 0.97 rms.
// The algorithms are those of Dekker (1971) and Knuth (the error-free sum).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "fp64_math.cuh"

namespace splash {
namespace f64 {

struct Pair {
  float h, l;
};

SPLASH_HD float float_of_bits(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float x;
  std::memcpy(&x, &b, 4);
  return x;
#endif
}
SPLASH_HD uint32_t float_bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t b;
  std::memcpy(&b, &x, 4);
  return b;
#endif
}
SPLASH_HD float fast_recip(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}
SPLASH_HD int exponent_field(double x) { return (int)((bits_of(x) >> 52) & 0x7ff); }

// h + l with |h| >= |l|
SPLASH_HD Pair pair_norm(float h, float l) {
  const float s = h + l;
  return Pair{s, l - (s - h)};
}
// x 2^(1023 - e0) as a pair (integer operations but for the remainder's
// scaling); false above 2^60 (and p without meaning); 0 below 2^-70
SPLASH_HD bool to_pair(double x, int e0, Pair& p) {
  const uint64_t b = bits_of(x);
  const int s = exponent_field(x) - e0;
  if (s > 60) return false;
  const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
  const uint32_t h = sign | ((uint32_t)(s + 127) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu);
  const float l = (float)((uint32_t)b & 0x1fffffffu) * float_of_bits((uint32_t)(s + 75) << 23);
  p = pair_norm(float_of_bits(h), float_of_bits(float_bits(l) ^ sign));
  if (s < -70) p = Pair{0.0f, 0.0f};
  return true;
}
// a float exactly, without a conversion instruction (0 for subnormals)
SPLASH_HD double widen(float x) {
  const uint32_t b = float_bits(x);
  if ((b & 0x7f800000u) == 0) return 0.0;
  const uint32_t hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20));
  return from_bits(((uint64_t)hi << 32) | (uint64_t)(b << 29));
}

SPLASH_HD Pair pair_add(const Pair& a, const Pair& b) {
  const float s = a.h + b.h, t = s - a.h;
  return pair_norm(s, ((a.h - (s - t)) + (b.h - t)) + (a.l + b.l));
}
SPLASH_HD Pair pair_neg(const Pair& a) { return Pair{-a.h, -a.l}; }
SPLASH_HD Pair pair_mul(const Pair& a, const Pair& b) {
  const float p = a.h * b.h;
  return pair_norm(p, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -p))));
}
// n / d given y = fast_recip(d.h): two corrections by the remainder, the first
// remainder as a pair
SPLASH_HD Pair pair_div(const Pair& n, const Pair& d, float y) {
  const float q = n.h * y;
  const float a = fmaf(-q, d.h, n.h), b = fmaf(-q, d.l, n.l);  // a is exact
  const float r = a + b, t = r - a;
  const float rl = (a - (r - t)) + (b - t);
  const float q1 = r * y;
  const float r2 = fmaf(-q1, d.l, fmaf(-q1, d.h, r) + rl);
  return pair_norm(q, fmaf(r2, y, q1));
}
// of pairs that pair_norm has made
SPLASH_HD bool pair_less(const Pair& a, const Pair& b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }

// What one side's limiter shares over the fields (LimiterLine): eta_plus,
// the superbee scale and the slope of the third-order line.
struct PairLine {
  Pair eta, sb, ts;
  bool ok;  // the Courant factor is positive and everything within range
};
// The largest superbee scale, a power of two.  limiter_pair takes ratios below
// 2^-70 for 0; a scale of 2^kMostScale makes 2^-50 of them, below the pairs'
// own error.  (Told apart per field instead of per side: hex(7) 3.35 -> 3.46 ms
// for 4 steps, quad(8) 2.92 -> 3.09 for 3.)
constexpr int kMostScale = 20;
SPLASH_HD PairLine pair_line(double eta_p, double sbs, double nu) {
  PairLine l;
  Pair n, s;
  const uint64_t nb = bits_of(nu);
  l.ok = (int64_t)nb > 0 && exponent_field(sbs) - exponent_field(nu) < kMostScale && to_pair(nu, 1023, n);
  l.ok = l.ok && to_pair(sbs, 1023, s) && to_pair(eta_p, 1023, l.eta) && s.h > 0.0f && l.eta.h > 0.0f;
  if (!l.ok) return l;
  l.sb = pair_div(s, n, fast_recip(n.h));
  // (1 + nu) / 3, 1/3 = 0x1.555556p-2 - 0x1.555556p-27
  l.ts = pair_mul(pair_add(Pair{1.0f, 0.0f}, n), Pair{0x1.555556p-2f, -0x1.555556p-27f});
  return l;
}

#if defined(SPLASH_SWITCH_TABLE)
// c + p d; the sum loses bits only where c is far below p d, whose weight in
// the switch is small then
SPLASH_HD Pair switch_term(const Pair& c, const Pair& p, const Pair& d) {
  const float m = p.h * d.h;
  const float ml = fmaf(p.h, d.h, -m) + fmaf(p.h, d.l, p.l * d.h);
  const float s = c.h + m, z = s - c.h;
  return Pair{s, ((c.h - (s - z)) + (m - z)) + (c.l + ml)};
}
// The switch h(r), r > 0 and not within 2^-40 below 1, from r and t = 1 - r
// (the rows of limiter_table.py).
SPLASH_HD Pair switch_pair(const Pair& r, const Pair& t) {
  const uint32_t rb = float_bits(r.h);
  if (rb >= 0x40100000u) return Pair{1.0f, 0.0f};  // r >= 2.25
  const bool above = t.h <= 0.0f;
  const uint32_t b = above ? (rb < 0x3f800000u ? 0x3f800000u : rb) : float_bits(t.h);
  int row;
  Pair d;
  if (above) {
    // the offset is (r - 1) - (centre - 1): t carries r - 1 without the
    // rounding of r
    row = (int)(b >> 15) - ((127 << 8) - 1280);
    d = pair_norm(-t.h - (float_of_bits(((b >> 15) << 15) | 0x4000u) - 1.0f), -t.l);
  } else {
    // t scaled to [1, 2) and its offset from the centre there; t = 1 is the
    // end of the last interval
    const bool one = b >= 0x3f800000u;
    row = one ? 1279 : (int)(b >> 18) - (87 << 5);
    const float up = float_of_bits((254u - (b >> 23) + (one ? 1u : 0u)) << 23);
    const float m = one ? 2.0f : float_of_bits((b & 0x7fffffu) | 0x3f800000u);
    const float c0 = one ? 1.984375f : float_of_bits(((b & 0x7c0000u) | 0x3f820000u));
    d = pair_norm(m - c0, t.l * up);
  }
#if defined(__CUDA_ARCH__)
  const float4* c = reinterpret_cast<const float4*>(kSwitchPairs[row]);
  const float4 a = __ldg(c), e = __ldg(c + 1), f = __ldg(c + 2);
#else
  struct {
    float x, y, z, w;
  } a, e, f;
  std::memcpy(&a, kSwitchPairs[row], 16);
  std::memcpy(&e, kSwitchPairs[row] + 4, 16);
  std::memcpy(&f, kSwitchPairs[row] + 8, 16);
#endif
  // c4 .. c7 in floats, then c3, c2, c1, c0 + d (...) in pairs
  const float q = fmaf(fmaf(fmaf(f.w, d.h, f.z), d.h, f.y), d.h, f.x);
  const Pair p3 = switch_term(Pair{e.z, e.w}, Pair{q, 0.0f}, d);
  const Pair p2 = switch_term(Pair{e.x, e.y}, p3, d);
  const Pair p1 = switch_term(Pair{a.z, a.w}, p2, d);
  const float m0 = p1.h * d.h;
  const float m0l = fmaf(p1.h, d.h, -m0) + fmaf(p1.h, d.l, p1.l * d.h);
  const float s0 = a.x + m0, z = s0 - a.x;
  return pair_norm(s0, (((a.x - (s0 - z)) + (m0 - z)) + a.y) + m0l);
}

// Whether limiter_pair serves these differences (for a PairLine that is ok):
// r no more than 2^59, and not within 2^-39 below 1.
SPLASH_HD bool pair_range(double dp, double num) {
  const int e0 = exponent_field(dp);
  if (e0 == 0 || e0 == 0x7ff || exponent_field(num) - e0 > 59) return false;
  // of like signs, the distance in units of the last place
  const uint64_t below = bits_of(dp) - bits_of(num);
  return below - 1 >= (1ull << 13) || ((bits_of(dp) ^ bits_of(num)) >> 63);
}

// The limiter of one field from dp, num = hr dm (r = num / dp) and
// e = dp - num (1 - r = e / dp); false where pairs do not serve.  hp receives
// the switch where it is needed.
SPLASH_HD bool limiter_pair(double dp, double num, double e, const PairLine& l, double& lim, Pair& hp) {
  if (!l.ok || !pair_range(dp, num)) return false;
  const int e0 = exponent_field(dp);
  Pair D, N, E;
  to_pair(dp, e0, D);
  to_pair(num, e0, N);
  to_pair(e, e0, E);
  // r <= 0, or below 2^-70: the limiter is 0, or taken for it (kMostScale)
  if (((bits_of(dp) ^ bits_of(num)) >> 63) || N.h == 0.0f) {
    lim = 0.0;
    return true;
  }
  const float y = fast_recip(D.h);
  const Pair r = pair_div(N, D, y), t = pair_div(E, D, y);
  const Pair one{1.0f, 0.0f};
  const Pair rs = pair_mul(r, l.sb);
  const Pair A = pair_less(rs, one) ? rs : one;
  const Pair B = pair_less(l.eta, r) ? l.eta : r;
  const Pair S = pair_less(A, B) ? B : A;
  Pair T = pair_add(one, pair_neg(pair_mul(l.ts, t)));
  Pair v = S;
  if (pair_less(T, S)) {
    if (T.h < 0.0f) T = Pair{0.0f, 0.0f};
    hp = switch_pair(r, t);
    v = pair_add(T, pair_mul(hp, pair_add(S, pair_neg(T))));
  }
  lim = widen(v.h) + widen(v.l);
  return true;
}
SPLASH_HD bool limiter_pair(double dp, double num, double e, const PairLine& l, double& lim) {
  Pair hp;
  return limiter_pair(dp, num, e, l, lim, hp);
}
#endif

// whether the difference dpg = dp BM / H+ is below 2^-8 of the scale with
// exponent field es
SPLASH_HD bool shallow(double dpg, int es) { return exponent_field(dpg) + 9 <= es; }

}  // namespace f64
}  // namespace splash
