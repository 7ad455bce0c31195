// integrands.cuh -- built-in integrand families as device functors.
//
// Each functor is templated on the dimension N and evaluates f(x) for a
// point x held in registers (double x[N]).  The families are Genz's test
// families (the ones the reference's drivers draw from, function.cu:70-214,
// and the north-star configurations) plus the reference driver's own
// cosine-sum integrand (cudaCuhre.cu:9-23).
//
// Parameters travel as GenzParams (one per integral); load() turns them
// into the functor's register form, folding constant work (a^2, a^-2).
//
// Axis products.  A functor whose value is a product of one factor per axis
// (Gaussian, product peak) says so with kAxisProduct, and the
// thread-per-region evaluator (axis_product_sums, region_rule.cuh) then
// forms the rule's set sums from per-axis factors.  It provides
//   axis(i)         axis i's parameters (also from a parameter block,
//                   axis_of), whose term(x) is what the axis contributes at x,
//   start(), step(acc, t), finish(acc)   the value as a left-to-right fold
//                   of the terms: operator() is that fold, so values formed
//                   either way have the same bits,
//   factor(t)       the axis' factor of the value,
//   factor2(t, s)   factor(t) + factor(s),
//   inverse(t, c)   1 / c for the factor c of term t,
//   noise(f0)       a bound of the rounding errors, relative to the values,
//                   by which a difference of fold values near f0 and the same
//                   difference formed from factors can disagree; three times
//                   what the operations can add up to.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include "rule9.hpp"

namespace cubature {

// Family identifiers (shared with the C ABI, include/cubature.h).
enum Family : int {
  kGaussian = 1,
  kOscillatory = 2,
  kCornerPeak = 3,
  kProductPeak = 4,
  kContinuous = 5,
  kDiscontinuous = 6,
  kCosSum = 7,
};

struct GenzParams {
  double a[kMaxDim];
  double u[kMaxDim];
};

// exp(-sum a_i^2 (x_i - u_i)^2)
template <int N>
struct Gaussian {
  double a[N], u[N];
  __host__ __device__ static Gaussian load(const GenzParams& p) {
    Gaussian g;
#pragma unroll
    for (int i = 0; i < N; ++i) { g.a[i] = p.a[i]; g.u[i] = p.u[i]; }
    return g;
  }
  static constexpr bool kAxisProduct = true;
  struct Axis {
    double a, u;
    __device__ __forceinline__ double term(double x) const { return a * (x - u); }
  };
  __device__ __forceinline__ static Axis axis_of(const GenzParams& p, int i) {
    return {p.a[i], p.u[i]};
  }
  __device__ __forceinline__ Axis axis(int i) const { return {a[i], u[i]}; }
  __device__ __forceinline__ static double start() { return 0.0; }
  __device__ __forceinline__ static double step(double s, double t) { return fma(t, t, s); }
  __device__ __forceinline__ static double finish(double s) { return exp(-s); }
  // exp(-t^2) with the rounding of t^2 corrected: a factor's error enters
  // many points alike, and does not average out as the points' own do
  __device__ __forceinline__ static double factor(double t) {
    const double tt = t * t;
    const double y = exp(-tt);
    return y > 0 ? fma(-fma(t, t, -tt), y, y) : y;
  }
  __device__ __forceinline__ static double factor2(double t, double s) {
    return factor(t) + factor(s);
  }
  __device__ __forceinline__ static double inverse(double, double c) { return 1 / c; }
  // The exponent s of a value v = exp(-s) is summed in N roundings of at most
  // s u (u = 2^-53) each, and v s is largest at the centre's s or below 1 / e;
  // 8 u for the exponentials, sums and quotients.
  __device__ __forceinline__ static double noise(double f0) {
    const int e = (__double2hiint(f0) >> 20) & 0x7ff;  // f0 >= 2^(e - 1023)
    const double s0 = e < 1022 ? 0.7 * (1023 - e) : 1.0;
    return 3.4e-16 * (N * s0 + 8);
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = start();
#pragma unroll
    for (int i = 0; i < N; ++i) s = step(s, axis(i).term(x[i]));
    return finish(s);
  }
};

// cos(2 pi u_0 + sum a_i x_i)
template <int N>
struct Oscillatory {
  double a[N], phase;
  __host__ __device__ static Oscillatory load(const GenzParams& p) {
    Oscillatory o;
#pragma unroll
    for (int i = 0; i < N; ++i) o.a[i] = p.a[i];
    o.phase = 2 * CUDART_PI * p.u[0];
    return o;
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = phase;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i] * x[i];
    return cos(s);
  }
};

// (1 + sum a_i x_i)^-(N+1)
template <int N>
struct CornerPeak {
  double a[N];
  __host__ __device__ static CornerPeak load(const GenzParams& p) {
    CornerPeak c;
#pragma unroll
    for (int i = 0; i < N; ++i) c.a[i] = p.a[i];
    return c;
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = 1;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i] * x[i];
    double p = 1;
#pragma unroll
    for (int k = 0; k <= N; ++k) p *= s;
    return 1 / p;
  }
};

// prod 1/(a_i^-2 + (x_i - u_i)^2)
template <int N>
struct ProductPeak {
  double ia2[N], u[N];
  __host__ __device__ static ProductPeak load(const GenzParams& p) {
    ProductPeak q;
#pragma unroll
    for (int i = 0; i < N; ++i) { q.ia2[i] = 1 / (p.a[i] * p.a[i]); q.u[i] = p.u[i]; }
    return q;
  }
  static constexpr bool kAxisProduct = true;
  struct Axis {
    double ia2, u;
    __device__ __forceinline__ double term(double x) const {
      const double t = x - u;
      return fma(t, t, ia2);
    }
  };
  __device__ __forceinline__ static Axis axis_of(const GenzParams& p, int i) {
    return {1 / (p.a[i] * p.a[i]), p.u[i]};
  }
  __device__ __forceinline__ Axis axis(int i) const { return {ia2[i], u[i]}; }
  __device__ __forceinline__ static double start() { return 1.0; }
  __device__ __forceinline__ static double step(double den, double q) { return den * q; }
  __device__ __forceinline__ static double finish(double den) { return 1 / den; }
  __device__ __forceinline__ static double factor(double q) { return 1 / q; }
  // 1/q + 1/p as (q + p) / (q p) with the roundings of the sum, the product
  // and the quotient corrected (a factor's error enters many points alike);
  // two divisions where the product leaves the normal range (a double's
  // biased exponent is in its high word's top bits)
  __device__ __forceinline__ static double factor2(double q, double p) {
    const double qp = q * p;
    const unsigned e = (unsigned)__double2hiint(qp) >> 20;
    if (e - 128u < 1791u) {
      const double s = q + p, b = s - q;
      const double es = (q - (s - b)) + (p - b), ep = fma(q, p, -qp);
      const double r = __drcp_rn(qp), y = s * r;
      return fma(fma(-y, ep, fma(-y, qp, s) + es), r, y);
    }
    return 1 / q + 1 / p;
  }
  __device__ __forceinline__ static double inverse(double q, double) { return q; }
  // N roundings of the product and the quotient, 8 of sums and factors; the
  // terms are the same bits on both sides
  __device__ __forceinline__ static double noise(double) { return 3.4e-16 * (N + 8); }
  __device__ __forceinline__ double operator()(const double* x) const {
    double den = start();
#pragma unroll
    for (int i = 0; i < N; ++i) den = step(den, axis(i).term(x[i]));
    return finish(den);
  }
};

// exp(-sum a_i |x_i - u_i|)
template <int N>
struct Continuous {
  double a[N], u[N];
  __host__ __device__ static Continuous load(const GenzParams& p) {
    Continuous c;
#pragma unroll
    for (int i = 0; i < N; ++i) { c.a[i] = p.a[i]; c.u[i] = p.u[i]; }
    return c;
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i] * fabs(x[i] - u[i]);
    return exp(-s);
  }
};

// 0 if x_0 > u_0 or x_1 > u_1, else exp(sum a_i x_i)
template <int N>
struct Discontinuous {
  double a[N], u0, u1;
  __host__ __device__ static Discontinuous load(const GenzParams& p) {
    Discontinuous c;
#pragma unroll
    for (int i = 0; i < N; ++i) c.a[i] = p.a[i];
    c.u0 = p.u[0];
    c.u1 = N > 1 ? p.u[1] : 2.0;
    return c;
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) s += a[i] * x[i];
    const bool out = x[0] > u0 || (N > 1 && x[N > 1 ? 1 : 0] > u1);
    return out ? 0.0 : exp(s);
  }
};

// -sum cos(10 x_i) / 0.054402111088937 / 2   (cudaCuhre.cu:11-22)
template <int N>
struct CosSum {
  __host__ __device__ static CosSum load(const GenzParams&) { return CosSum(); }
  __device__ __forceinline__ double operator()(const double* x) const {
    double s = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) s = s - cos(10.0 * x[i]) / 0.054402111088937;
    return s / 2.0;
  }
};

// One integrand of any built-in family, chosen per integral: the family's
// functor is built once (per region, by the source) and called point by point.
// Single-family batches sum the factored families from factors on long lists
// and products in the second phase, so a mixed batch agrees with them to
// rounding there (the points' values are the same).
template <int N>
struct MixedGenz {
  int family;
  union {
    Gaussian<N> g;
    Oscillatory<N> o;
    CornerPeak<N> c;
    ProductPeak<N> p;
    Continuous<N> ct;
    Discontinuous<N> d;
  } f;
  __host__ __device__ static MixedGenz make(const GenzParams& q, int family) {
    MixedGenz m;
    m.family = family;
    switch (family) {
      case kGaussian: m.f.g = Gaussian<N>::load(q); break;
      case kOscillatory: m.f.o = Oscillatory<N>::load(q); break;
      case kCornerPeak: m.f.c = CornerPeak<N>::load(q); break;
      case kProductPeak: m.f.p = ProductPeak<N>::load(q); break;
      case kContinuous: m.f.ct = Continuous<N>::load(q); break;
      case kDiscontinuous: m.f.d = Discontinuous<N>::load(q); break;
      default: break;
    }
    return m;
  }
  __device__ __forceinline__ double operator()(const double* x) const {
    switch (family) {
      case kGaussian: return f.g(x);
      case kOscillatory: return f.o(x);
      case kCornerPeak: return f.c(x);
      case kProductPeak: return f.p(x);
      case kContinuous: return f.ct(x);
      case kDiscontinuous: return f.d(x);
      default: return CosSum<N>()(x);
    }
  }
};

}  // namespace cubature
