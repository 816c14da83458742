// Arithmetic of the FP64 path, written for a narrow FP64 pipe.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles (8.16 ns
// measured from 4 warps per SM on, 2 thread operations per SM and cycle, FMA,
// add, multiply and compare alike, 1/64 of FP32), one per scheduler every 33
// ns, whether it depends on the last or not.  So the FP64 kernels' time is the
// number of FP64 instructions; what else issues beside them is nearly free.
// Hence
//   * multiply-adds are written as fma explicitly (these files are compiled
//     with -fmad=false, so nothing else is fused and the scalar types below
//     agree to the last bit),
//   * a quotient is the hardware's reciprocal seed (rcp.approx.ftz.f64,
//     2^-19.9, on the special-function unit), one third-order Newton step
//     (Householder's method) and, where the quotient itself is kept, the
//     residual correction of Markstein (1990): 4 or 6 instructions; a root
//     is the same from rsqrt.approx.ftz.f64 (2^-20.0).  Operands or quotients
//     that are subnormal, infinite, NaN or next to the ends of the range leave
//     through integer tests to the exact operator, so those give what it gives,
//   * comparisons are integer comparisons of the bit patterns.
// Every function is a template over the scalar: double, Dual<N> (values by
// the same operations, derivatives by the chain rule) and Taped (taped.cuh).
// On the host the plain operators stand in for the seeds.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "dual.cuh"

namespace splash {
namespace f64 {

// ---- scalars ------------------------------------------------------------
template <class A, class B, class C = double>
using wider_t = std::conditional_t<!std::is_same<A, double>::value, A,
                                   std::conditional_t<!std::is_same<B, double>::value, B, C>>;

SPLASH_HD uint64_t bits_of(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
SPLASH_HD double from_bits(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
SPLASH_HD uint32_t high_word(double x) { return (uint32_t)(bits_of(x) >> 32); }

// a b + c with one rounding; the derivative skips operands without tangents
template <class A, class B, class C>
SPLASH_HD wider_t<A, B, C> fm(const A& a, const B& b, const C& c) {
  using R = wider_t<A, B, C>;
  if constexpr (std::is_same<R, double>::value) {
    return ::fma(a, b, c);
  } else {
    R r(::fma(val(a), val(b), val(c)));
    if constexpr (is_dual<R>::value) {
#pragma unroll
      for (int i = 0; i < R::kN; ++i) {
        double t = 0.0;
        if constexpr (is_dual<C>::value) t = c.d[i];
        if constexpr (is_dual<A>::value) t = is_dual<C>::value ? ::fma(a.d[i], val(b), t) : a.d[i] * val(b);
        if constexpr (is_dual<B>::value)
          t = (is_dual<A>::value || is_dual<C>::value) ? ::fma(val(a), b.d[i], t) : val(a) * b.d[i];
        r.d[i] = t;
      }
    }
    return r;
  }
}

// ---- comparisons --------------------------------------------------------
SPLASH_HD bool nan_bits(double x) { return (bits_of(x) << 1) > 0xffe0000000000000ull; }
// NaN or infinite
SPLASH_HD bool odd_bits(double x) { return (high_word(x) & 0x7ff00000u) == 0x7ff00000u; }
// the order of the reals as the order of signed integers
SPLASH_HD int64_t order_key(double x) {
  const int64_t b = (int64_t)bits_of(x);
  return b ^ (int64_t)((uint64_t)(b >> 63) >> 1);
}
// a < b as integers, false with a NaN like the operator (-0 orders below +0)
SPLASH_HD bool less(double a, double b) {
#if defined(__CUDA_ARCH__)
  return order_key(a) < order_key(b) && !nan_bits(a) && !nan_bits(b);
#else
  return a < b;
#endif
}
template <class T>
SPLASH_HD bool less(const T& a, const T& b) {
  if constexpr (is_dual<T>::value)
    return less(a.v, b.v);
  else
    return a < b;
}
// a < b of two non-negative numbers, neither NaN
SPLASH_HD bool less_pos(double a, double b) {
#if defined(__CUDA_ARCH__)
  return bits_of(a) < bits_of(b);
#else
  return a < b;
#endif
}
// comparisons with zero, false with a NaN
SPLASH_HD bool not_below_zero(double x) {
  const int64_t b = (int64_t)bits_of(x);
  return b >= 0 ? b <= 0x7ff0000000000000ll : b == INT64_MIN;
}
SPLASH_HD bool below_zero(double x) {
  const uint64_t b = bits_of(x);
  return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}
template <class T>
SPLASH_HD bool not_below_zero(const T& x) {
  if constexpr (is_dual<T>::value)
    return not_below_zero(x.v);
  else
    return x >= 0;
}
template <class T>
SPLASH_HD bool below_zero(const T& x) {
  if constexpr (is_dual<T>::value)
    return below_zero(x.v);
  else
    return x < 0;
}
// std::max / std::min argument semantics
template <class T>
SPLASH_HD T smax(const T& a, const T& b) {
  return less(a, b) ? b : a;
}
template <class T>
SPLASH_HD T smin(const T& a, const T& b) {
  return less(b, a) ? b : a;
}

// ---- reciprocal, quotient, root -----------------------------------------
// The exact operators, out of line: inlined they were evaluated on every
// path and selected from (478 instead of 250 FP64 instructions per side in
// the isothermal edge launch).
#if defined(__CUDA_ARCH__)
#define SPLASH_COLD static __device__ __noinline__
#else
#define SPLASH_COLD inline
#endif
SPLASH_COLD double exact_quotient(double a, double b) { return a / b; }
SPLASH_COLD double exact_root(double x) { return ::sqrt(x); }

// 1 / b to 1 ulp
SPLASH_HD double recip(double b) {
#if defined(__CUDA_ARCH__)
  // normal with a normal reciprocal: exponent field 2 .. 2044
  if ((high_word(b) & 0x7fffffffu) - 0x00200000u < 0x7fb00000u) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = ::fma(-b, y, 1.0);
    return ::fma(y, ::fma(e, e, e), y);
  }
#endif
  return exact_quotient(1.0, b);
}
// normal, and twice the smallest normal number or more
SPLASH_HD bool well_normal(double x) { return (high_word(x) & 0x7fffffffu) - 0x00200000u < 0x7fd00000u; }
// a / b given y = recip(b): Markstein's correction, the operator's bits.  It
// needs the remainder a - b q exactly, which holds from |a| = 2^-899 on (its
// last place is 2^-106 of a), and a quotient and a reciprocal with all their
// bits; the rest is the operator's.  Zeros, which quiet flows are full of, are
// a y, whose sign the correction would lose (-0 + 0).
SPLASH_HD double quotient(double a, double b, double y) {
#if defined(__CUDA_ARCH__)
  const double q = a * y;
  const double c = ::fma(::fma(-b, q, a), y, q);
  if (well_normal(y)) {
    if ((high_word(a) & 0x7fffffffu) >= 0x07c00000u && well_normal(c)) return c;
    if (bits_of(a) << 1 == 0) return q;
  }
#endif
  return exact_quotient(a, b);
}
// sqrt(x) to 1 ulp; `inv` receives 1 / sqrt(x)
SPLASH_HD double root_pair(double x, double& inv) {
#if defined(__CUDA_ARCH__)
  if (high_word(x) - 0x00200000u < 0x7fb00000u) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = x * y;
    const double e = ::fma(-h, y, 1.0);
    const double p = ::fma(e, 0.375, 0.5);
    inv = ::fma(y * e, p, y);
    return ::fma(p, h * e, h);
  }
#endif
  const double s = exact_root(x);
  inv = exact_quotient(1.0, s);
  return s;
}
SPLASH_HD double root(double x) {
  double inv;
  return root_pair(x, inv);
}

template <class T>
SPLASH_HD T recip(const T& b) {
  T r(recip(val(b)));
  if constexpr (is_dual<T>::value) {
    const double s = -r.v * r.v;
#pragma unroll
    for (int i = 0; i < T::kN; ++i) r.d[i] = s * b.d[i];
  }
  return r;
}
// a / b, rounded like the operator
template <class A, class B>
SPLASH_HD wider_t<A, B> divide(const A& a, const B& b) {
  using R = wider_t<A, B>;
  const double y = recip(val(b));
  R r(quotient(val(a), val(b), y));
  if constexpr (is_dual<R>::value) {
#pragma unroll
    for (int i = 0; i < R::kN; ++i) {
      double t = 0.0;
      if constexpr (is_dual<A>::value) t = a.d[i];
      if constexpr (is_dual<B>::value) t = is_dual<A>::value ? ::fma(-r.v, b.d[i], t) : -r.v * b.d[i];
      r.d[i] = t * y;
    }
  }
  return r;
}
template <class T>
SPLASH_HD T root(const T& x) {
  double inv;
  T r(root_pair(val(x), inv));
  if constexpr (is_dual<T>::value) {
    // at 0 (a zero velocity's norm) the one-sided derivative is taken as 0
    const double h = (r.v > 0.0) ? 0.5 * inv : 0.0;
#pragma unroll
    for (int i = 0; i < T::kN; ++i) r.d[i] = h * x.d[i];
  }
  return r;
}

// ---- the limiter's switch -----------------------------------------------
// h(r) of physics/adiabatic.hpp:692-702 through exact identities: for
// y, z >= 0, 1 - tanh(y) = 2 / (1 + e^{2y}) and tanh(z) = expm1(2z) /
// (expm1(2z) + 2), with 2z clamped at 80 (tanh(40) is 1 in double).
// `slope` receives dh/dr.
SPLASH_HD double switch_formula(double r, double& slope) {
  slope = 0.0;
  if (r < 1 && r > 0) {
    const double p = ::exp(0.1 * ::log(1 - r));
    const double h = 2 / (1 + ::exp(8 * (r * r) * p));
    slope = -h * (1 - h / 2) * (16 * r * p - 0.8 * (r * r) * p / (1 - r));
    return h;
  }
  if (r >= 1) {
    const double x = r - 1;
    const double em = ::expm1(fmin(20 * ((x * x) * x), 80.0));
    const double t = em / (em + 2);
    const double t2 = t * t;
    slope = 180 * ((t2 * t2) * t) * (1 - t2) * (x * x);
    return (t2 * t2) * t2;
  }
  return 0.0;
}

#if defined(SPLASH_SWITCH_TABLE)
#if defined(__CUDACC__)
#define SPLASH_TABLE __device__ __align__(64)
#else
#define SPLASH_TABLE static
#endif
#include "limiter_switch_table.inc"  // written by limiter_table.py at build time
#endif

#if defined(__CUDACC__) && defined(SPLASH_SWITCH_TABLE)
__device__ __forceinline__ double horner8(const double* __restrict__ row, double d) {
  const double2* c = reinterpret_cast<const double2*>(row);
  const double2 a = __ldg(c), b = __ldg(c + 1), e = __ldg(c + 2), f = __ldg(c + 3);
  return ::fma(::fma(::fma(::fma(::fma(::fma(::fma(f.y, d, f.x), d, e.y), d, e.x), d, b.y), d, b.x), d, a.y), d, a.x);
}
// The row of r > 0 and the offset from its centre; row -1: 1 - r below
// 2^-40 or past the table (limiter_table.py describes the intervals).
__device__ __forceinline__ int switch_row(double r, double& d) {
  const uint32_t hr = high_word(r);
  const bool above = hr >= 0x3ff00000u;
  const double u = above ? r : 1 - r;
  const uint32_t hu = high_word(u);
  const int sh = above ? 12 : 15;
  int row = (int)(hu >> sh) - (above ? (1023 << 8) - 1280 : 983 << 5);
  uint32_t mid = ((hu >> sh) << sh) | (1u << (sh - 1));
  if (!above && hu == 0x3ff00000u) {  // u = 1: the end of the last interval
    row = 1279;
    mid = 0x3fefc000u;
  }
  d = u - __hiloint2double((int)mid, 0);
  return (above ? row < 1568 : row >= 0) ? row : -1;
}
#endif

// h(r) for r > 0 (not NaN) and dh/dr; with `known`, h comes in and only the
// slope is evaluated
SPLASH_HD double switch_slope(double r, bool known, double h, double& slope) {
#if defined(__CUDA_ARCH__) && defined(SPLASH_SWITCH_TABLE)
  slope = 0.0;
  if (high_word(r) >= 0x40020000u) return 1.0;  // r >= 2.25
  double d;
  const int row = switch_row(r, d);
  if (row >= 0) {
    slope = horner8(kSwitchSlope[row], d);
    return known ? h : horner8(kSwitchTable[row], d);
  }
#endif
  return switch_formula(r, slope);
}
SPLASH_HD double switch_pos(double r) {
#if defined(__CUDA_ARCH__) && defined(SPLASH_SWITCH_TABLE)
  if (high_word(r) >= 0x40020000u) return 1.0;
  double d;
  const int row = switch_row(r, d);
  if (row >= 0) return horner8(kSwitchTable[row], d);
#endif
  double slope;
  return switch_formula(r, slope);
}

// 1 - h^M with h = min(a / b, b / a) for a, b > 0 (the pressure switch of
// HLLCplus.hpp).  Near h = 1, where 1 - h^M cancels, through
// log h = -2 atanh s, s = |a - b| / (a + b) < 2^-6, and the series of
// expm1; the truncations are below 2^-58 of the result.
template <class T>
SPLASH_HD T pressure_switch(const T& M, const T& a, const T& b) {
  const T diff = a - b;
  T s = divide(diff, a + b);
  const bool flip = (bits_of(val(s)) >> 63) != 0;
  if (flip) s = -s;
  if (less_pos(val(s), 0.015625)) {
    const double x = val(s), m = val(M);
    const double x2 = x * x;
    const double at = ::fma(x2, ::fma(x2, ::fma(x2, ::fma(x2, 1.0 / 9, 1.0 / 7), 1.0 / 5), 1.0 / 3), 1.0);
    const double L = -2 * x * at;  // log h
    const double y = m * L;
    double q = ::fma(y, 1.0 / 40320, 1.0 / 5040);
    q = ::fma(y, q, 1.0 / 720);
    q = ::fma(y, q, 1.0 / 120);
    q = ::fma(y, q, 1.0 / 24);
    q = ::fma(y, q, 1.0 / 6);
    q = ::fma(y, q, 0.5);
    q = ::fma(y, q, 1.0);
    T g(-y * q);
    if constexpr (is_dual<T>::value) {
      const double E = 1 - g.v;  // h^M
      const double dm = -E * L, ds = E * m * 2 * recip(1 - x2);
#pragma unroll
      for (int i = 0; i < T::kN; ++i) g.d[i] = ::fma(dm, M.d[i], ds * s.d[i]);
    }
    return g;
  }
  const double pa = val(a), pb = val(b);
  const double hA = pa / pb, hB = pb / pa;
  const bool second = hB < hA;
  const double h = second ? hB : hA;
  const double L = ::log(h);
  const double E = ::exp(val(M) * L);
  T g(1 - E);
  if constexpr (is_dual<T>::value) {
    // log h = +-(log a - log b)
    const double sg = second ? -1.0 : 1.0;
    const double ia = sg / pa, ib = sg / pb;
#pragma unroll
    for (int i = 0; i < T::kN; ++i)
      g.d[i] = -E * ::fma(L, M.d[i], val(M) * (ia * a.d[i] - ib * b.d[i]));
  }
  return g;
}

}  // namespace f64
}  // namespace splash
