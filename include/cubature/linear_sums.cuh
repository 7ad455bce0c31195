// linear_sums.cuh -- the rule's set sums over one region by one thread
// (ThreadSums, region_rule.cuh) for corner peak and continuous.
//
// A rule point lies at the box's centre plus or minus g H_d on each axis d it
// moves, and every set holds both signs of every move.
//   corner peak   with the argument b at the centre and increments
//                 t_d = a_d g H_d the points pair up as (b + s)^-(N+1) +
//                 (b - s)^-(N+1), one division per pair;
//   continuous    a product over the axes, exp(-a_d |x_d - u_d|) each.
// The split axis comes from these sums where they tell the axes apart by more
// than the rounding, else from the points (exact_axis_points).
//
// Oscillatory would factor too (2 cos b cos t per pair of points, 18 to 37
// times faster) and more exactly, but is evaluated point by point: where it is
// smooth over a small region the error estimate is nothing but the rounding of
// the points, and the exact form would change such estimates by about 1e-9 of
// the value, and with them which regions are finished at tolerances that low.
#pragma once

#include "integrands.cuh"
#include "region_rule.cuh"

namespace cubature {
namespace detail {

constexpr double kRound3 = 3.4e-16;  // three units of rounding (2^-53), rounded up

// b += a x, with what the rounding of the product and the sum leaves out
// added to lo: an error of the centre's argument is shared by all points of
// the region and does not average out as the points' own do.  (Intrinsics: a
// contraction of the residual's terms would count the product's rounding
// twice.)
__device__ __forceinline__ void add_product(double& b, double& lo, double a, double x) {
  const double p = __dmul_rn(a, x), s = __dadd_rn(b, p), v = __dadd_rn(s, -b);
  const double rest = __dadd_rn(__dadd_rn(b, -__dadd_rn(s, -v)), __dadd_rn(p, -v));
  lo = __dadd_rn(lo, __dadd_rn(fma(a, x, -p), rest));
  b = s;
}

// s^M by squaring.
template <int M>
__device__ __forceinline__ double int_power(double s) {
  if constexpr (M == 1) {
    return s;
  } else if constexpr (M % 2 == 0) {
    const double h = int_power<M / 2>(s);
    return h * h;
  } else {
    return s * int_power<M - 1>(s);
  }
}

// 552 pairs of about 23 FP64 instructions in 8 dimensions instead of 1105
// points of 35: a chain of 78 us for one thread (33 us in 6, 13 us in 4
// dimensions), so 32 lanes point by point are faster for short lists (8-D:
// 51 us for 8192 regions, 192 us for 32 768).
template <int N>
struct ThreadSums<CornerPeak<N>> {
  static constexpr bool value = true;
  static constexpr int kMinList = 2048 * (N - 2);
  // An argument beyond the range of a double becomes the largest one: a point's
  // value is 0 either way, and the difference of two infinities is no number.
  __device__ __forceinline__ static double finite(double x) {
    constexpr double kMax = 1.7976931348623157e308;
    return fabs(x) > kMax ? copysign(kMax, x) : x;
  }
  // (b + s)^-(N+1) + (b - s)^-(N+1); two divisions where the product of the
  // powers leaves the normal range
  __device__ __forceinline__ static double pair(double b, double s) {
    const double p = int_power<N + 1>(b + s), q = int_power<N + 1>(b - s), pq = p * q;
    const unsigned e = ((unsigned)__double2hiint(pq) >> 20) & 0x7ffu;
    return e - 64u < 1919u ? (p + q) / pq : 1 / p + 1 / q;
  }
  __device__ __forceinline__ static void run(const CornerPeak<N>& f, const double (&L)[N],
                                             const double (&H)[N], double ratio, RegionSums& out) {
    double b = 1, lo = 0, mag = 1, top = 0, t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      add_product(b, lo, f.a[i], fma(0.5, H[i], L[i]));
      mag += fabs(f.a[i]) * fmax(fabs(L[i]), fabs(L[i] + H[i]));
      t[i] = finite(f.a[i] * H[i]);
      top = fmax(top, fabs(t[i]));
    }
    if (finite(b) != b) {
      b = finite(b);
      lo = 0;
    }
    const double f0 = 1 / int_power<N + 1>(b);
    double S1 = 0, S2 = 0, S3 = 0, S4 = 0, S5 = 0, S6 = 0, S7 = 0, S8 = 0;
    AxisChoice ch;
#pragma unroll 1
    for (int d = 0; d < N; ++d) {
      const double s = pair(b, kGenA1 * t[d]), w = pair(b, kGenA2 * t[d]);
      ch.add(d, 1.0, fabs(f0), f0 < 0 ? -s : s, f0 < 0 ? -w : w, ratio);
      S1 += s;
      S2 += w;
      S3 += pair(b, kGenA3 * t[d]);
      S4 += pair(b, kGenA4 * t[d]);
      const double td = kGenA1 * t[d];
#pragma unroll 1
      for (int e = 0; e < N; ++e) {
        if (e == d) continue;
        S6 += pair(b, fma(kGenA2, t[e], td)) + pair(b, fma(-kGenA2, t[e], td));
        if (e < d) continue;
        const double p = fma(kGenA1, t[e], td), m = fma(-kGenA1, t[e], td);
        S5 += pair(b, p) + pair(b, m);
#pragma unroll 1
        for (int g = e + 1; g < N; ++g) {
          const double tg = kGenA1 * t[g];
          S7 += (pair(b, p + tg) + pair(b, p - tg)) + (pair(b, m + tg) + pair(b, m - tg));
        }
      }
    }
    // the corners: axis 0's sign fixed (a pair holds both), the last two axes'
    // signs side by side
    constexpr int kHigh = N > 3 ? N - 3 : 0;
#pragma unroll 1
    for (int m = 0; m < (1 << kHigh); ++m) {
      double s = kGenL * t[0];
#pragma unroll
      for (int i = 0; i < kHigh; ++i) s = fma((m >> i) & 1 ? -kGenL : kGenL, t[1 + i], s);
      if constexpr (N == 2) {
        S8 += pair(b, fma(kGenL, t[1], s)) + pair(b, fma(-kGenL, t[1], s));
      } else {
        const double p = fma(kGenL, t[N - 2], s), q = fma(-kGenL, t[N - 2], s);
        const double l = kGenL * t[N - 1];
        S8 += (pair(b, p + l) + pair(b, p - l)) + (pair(b, q + l) + pair(b, q - l));
      }
    }
    // The argument's centre is b + lo: a relative change of -(N + 1) lo / b for
    // the centre, of -(N + 1) lo / (b + s) for a point.  Taken for all of them:
    // a point with a smaller argument keeps part of its error, one with a larger
    // argument is left with at most the centre's on a value below the centre's.
    const double corr = fma(-(N + 1.0) * lo, 1 / b, 1.0);
    out.S[0] = f0 * corr;
    out.S[1] = S1 * corr;
    out.S[2] = S2 * corr;
    out.S[3] = S3 * corr;
    out.S[4] = S4 * corr;
    out.S[5] = S5 * corr;
    out.S[6] = S6 * corr;
    out.S[7] = S7 * corr;
    out.S[8] = S8 * corr;
    out.best = ch.best;
    // a value's relative error: N + 1 times that of its argument (N roundings
    // of at most mag u, against an argument of at least `low`), and N + 1
    // roundings of the power
    const double low = fabs(b) - 0.5 * top;
    const bool sure = low > 0.1 * fabs(b) &&
                      ch.sure(kRound3 * ((N + 1) * (N * mag / low + 2) + 8), fabs(f0));
    out.axis = sure ? ch.axis : exact_axis_points<N>(f, L, H, ratio);
  }
};

// 11 N exponentials instead of one per point (for 2 dimensions 22 against 33).
//
// With coefficients of both signs a product of some axes' factors can leave
// the range of a double where the value does not; with exponents that add up to
// less than kRange over the box none does.  Beyond it (values of 1e260, or
// their reciprocals, inside one box) the region is evaluated point by point.
template <int N>
struct ThreadSums<Continuous<N>> {
  static constexpr bool value = true;
  static constexpr int kMinList = 0;
  static constexpr double kRange = 600;
  // noise0: the sum of an exponent's magnitudes where its terms have both
  // signs (kGrows)
  template <bool kGrows>
  __device__ __forceinline__ static void factored(const Continuous<N>& f, const double (&L)[N],
                                                  const double (&H)[N], double ratio,
                                                  double noise0, RegionSums& out) {
    AxisPoly poly;
    AxisChoice ch;
#pragma unroll 1
    for (int d = 0; d < N; ++d) {
      // exp(-a |x - u|) with the rounding of the product corrected
      auto factor = [&](double x) {
        const double v = fabs(x - f.u[d]), p = f.a[d] * v, y = exp(-p);
        return y > 0 ? fma(-fma(f.a[d], v, -p), y, y) : y;
      };
      auto at = [&](double gen, bool minus) { return factor(fma(coef(gen, minus), H[d], L[d])); };
      const double c = factor(fma(0.5, H[d], L[d]));
      const double s = at(kGenA1, false) + at(kGenA1, true);
      const double w = at(kGenA2, false) + at(kGenA2, true);
      ch.add(d, 1 / c, c, s, w, ratio);
      poly.append(c, s, w, at(kGenA3, false) + at(kGenA3, true),
                  at(kGenA4, false) + at(kGenA4, true), at(kGenL, false) + at(kGenL, true));
    }
    poly.store(out);
    out.best = ch.best;
    // as Gaussian::noise: the exponent of a value is summed in N roundings
    const int e = (__double2hiint(poly.z) >> 20) & 0x7ff;
    const double s0 = kGrows ? noise0 : e < 1022 ? 0.7 * (1023 - e) : 1.0;
    out.axis = ch.sure(kRound3 * (2 * N * s0 + 8), poly.z) ? ch.axis
                                                           : exact_axis_points<N>(f, L, H, ratio);
  }
  __device__ __noinline__ static void by_points(const Continuous<N>& f, const double (&L)[N],
                                                const double (&H)[N], double ratio,
                                                RegionSums& out) {
    ItemTable<N> tab;
    tab.fill();
    region_point_sums<N, 1>(f, L, H, 0, tab, ratio, out);
  }
  // Out of line: within run() it took 10 to 17% more time for the regions
  // without a growing axis (17.7 -> 20.7 us for 65 536 6-D ones), and so did sums
  // returned by value: more registers, fewer warps.
  __device__ __noinline__ static void growing(const Continuous<N>& f, const double (&L)[N],
                                              const double (&H)[N], double ratio,
                                              RegionSums& out) {
    double reach = 0;  // largest sum of the exponents' magnitudes
#pragma unroll
    for (int i = 0; i < N; ++i)
      reach = fma(fabs(f.a[i]), fmax(fabs(L[i] - f.u[i]), fabs(L[i] + H[i] - f.u[i])), reach);
    if (reach < kRange)
      factored<true>(f, L, H, ratio, reach, out);
    else
      by_points(f, L, H, ratio, out);
  }
  __device__ __forceinline__ static void run(const Continuous<N>& f, const double (&L)[N],
                                             const double (&H)[N], double ratio, RegionSums& out) {
    bool decays = true;
#pragma unroll
    for (int i = 0; i < N; ++i) decays = decays && f.a[i] >= 0;
    if (decays)
      factored<false>(f, L, H, ratio, 0, out);
    else
      growing(f, L, H, ratio, out);
  }
};

}  // namespace detail
}  // namespace cubature
