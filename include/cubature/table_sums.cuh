// table_sums.cuh -- the rule's set sums of the 7-D table integrand over one
// region by one thread (see ThreadSums, region_rule.cuh).
#pragma once

#include "region_rule.cuh"
#include "tables.cuh"

namespace cubature {
namespace detail {

// One region by one thread.  The integrand is a product over the axis
// groups {0}, {1, 2} and {3, 4, 5, 6}, and a rule point moves at most three
// axes (or all of them, the corners), so the 717 points need only 11
// spline values, 33 table cells and 153 kernel values: each group's sums
// over the patterns a set can have inside it, combined by the distributive
// law as in axis_product_sums.  The kernel's argument is linear in its
// axes, so its points are the centre's argument plus one increment per
// moved axis; the centre and the points of sets 1 and 2 are evaluated as
// operator() does (same bits), for the split axis.  The loops are kept
// rolled: unrolled, the body does not fit the instruction cache.
template <>
struct ThreadSums<Table7<7>> {
  static constexpr bool value = true;
  static constexpr int kMinList = 0;
  __device__ __forceinline__ static void run(const Table7<7>& f, const double (&L)[7], const double (&H)[7],
                                              double ratio, RegionSums& out) {
    auto kernel = [&](double r) { return f.kernel(r); };
    double C[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) C[i] = fma(0.5, H[i], L[i]);
    const double a0 = f.spline(C[0]), b0 = f.grid(C[1], C[2]);
    const double rc = f.kernel_arg(C[3], C[4], C[5], C[6]);
    const double c0 = kernel(rc), ab = a0 * b0;
    const double f0 = ab * c0;
    const double base = __dmul_rn(__dmul_rn(f0, 2.0), __dadd_rn(1.0, -ratio));
    double best = 0;
    int axis = -1;
    auto fourth_difference = [&](int d, double f1p, double f1m, double f2p, double f2m) {
      const double fd = fabs(__dadd_rn(__dadd_rn(base, __dmul_rn(ratio, __dadd_rn(f1p, f1m))),
                                       -__dadd_rn(f2p, f2m)));
      if (fd > best) {
        best = fd;
        axis = d;
      }
    };

    // axis 0: sums over +-g of the spline per generator
    double ea[5];
    {
      double v[4];
#pragma unroll 1
      for (int k = 0; k < 5; ++k) {
        const double g = k == 0 ? kGenA1 : k == 1 ? kGenA2 : k == 2 ? kGenA3 : k == 3 ? kGenA4 : kGenL;
        const double vp = f.spline(fma(coef(g, false), H[0], L[0]));
        const double vm = f.spline(fma(coef(g, true), H[0], L[0]));
        const double sum = vp + vm;
        if (k == 0) { v[0] = vp; v[1] = vm; ea[0] = sum; }
        if (k == 1) { v[2] = vp; v[3] = vm; ea[1] = sum; }
        if (k == 2) ea[2] = sum;
        if (k == 3) ea[3] = sum;
        if (k == 4) ea[4] = sum;
      }
      fourth_difference(0, v[0] * b0 * c0, v[1] * b0 * c0, v[2] * b0 * c0, v[3] * b0 * c0);
    }

    // axes 1 and 2: one axis moved (per generator a1..a4), both moved
    // (a1 a1, a1 a2 either way, corners)
    double eb[4] = {0, 0, 0, 0};
    double b11 = 0, b12 = 0, bl = 0;
#pragma unroll 1
    for (int d = 1; d <= 2; ++d) {
      const double Ld = d == 1 ? L[1] : L[2], Hd = d == 1 ? H[1] : H[2];
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double g = k < 2 ? kGenA1 : k < 4 ? kGenA2 : k < 6 ? kGenA3 : kGenA4;
        const double t = fma(coef(g, k & 1), Hd, Ld);
        v[k] = f.grid(d == 1 ? t : C[1], d == 1 ? C[2] : t);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) eb[k] += v[2 * k] + v[2 * k + 1];
      fourth_difference(d, a0 * v[0] * c0, a0 * v[1] * c0, a0 * v[2] * c0, a0 * v[3] * c0);
    }
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      const double g1 = k == 3 ? kGenL : k == 2 ? kGenA2 : kGenA1;
      const double g2 = k == 3 ? kGenL : k == 1 ? kGenA2 : kGenA1;
      double sum = 0;
#pragma unroll
      for (int s = 0; s < 4; ++s)
        sum += f.grid(fma(coef(g1, s & 1), H[1], L[1]), fma(coef(g2, s & 2), H[2], L[2]));
      if (k == 0) b11 = sum;
      else if (k == 3) bl = sum;
      else b12 += sum;
    }

    // axes 3 to 6: increments of the kernel's argument per unit generator
    const double w[4] = {4.0 * H[3], 2.0 * H[4], 0.1 * H[5], 0.1 * H[6]};
    double ec[4] = {0, 0, 0, 0};
    double c11 = 0, c12 = 0, c111 = 0, cl = 0;
#pragma unroll 1
    for (int d = 0; d < 4; ++d) {
      const double Ld = d == 0 ? L[3] : d == 1 ? L[4] : d == 2 ? L[5] : L[6];
      const double Hd = d == 0 ? H[3] : d == 1 ? H[4] : d == 2 ? H[5] : H[6];
      const double wd = d == 0 ? w[0] : d == 1 ? w[1] : d == 2 ? w[2] : w[3];
      double v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double t = fma(coef(k < 2 ? kGenA1 : kGenA2, k & 1), Hd, Ld);
        v[k] = kernel(f.kernel_arg(d == 0 ? t : C[3], d == 1 ? t : C[4], d == 2 ? t : C[5],
                                 d == 3 ? t : C[6]));
      }
      fourth_difference(d + 3, ab * v[0], ab * v[1], ab * v[2], ab * v[3]);
      ec[0] += v[0] + v[1];
      ec[1] += v[2] + v[3];
      ec[2] += kernel(fma(kGenA3, wd, rc)) + kernel(fma(-kGenA3, wd, rc));
      ec[3] += kernel(fma(kGenA4, wd, rc)) + kernel(fma(-kGenA4, wd, rc));
#pragma unroll 1
      for (int e = 0; e < 4; ++e) {
        if (e == d) continue;
        const double we = e == 0 ? w[0] : e == 1 ? w[1] : e == 2 ? w[2] : w[3];
        const double rp = fma(kGenA1, wd, rc), rm = fma(-kGenA1, wd, rc);
        c12 += (kernel(fma(kGenA2, we, rp)) + kernel(fma(-kGenA2, we, rp))) +
               (kernel(fma(kGenA2, we, rm)) + kernel(fma(-kGenA2, we, rm)));
        if (e < d) continue;
        const double r2[4] = {fma(kGenA1, we, rp), fma(-kGenA1, we, rp), fma(kGenA1, we, rm),
                              fma(-kGenA1, we, rm)};
        c11 += (kernel(r2[0]) + kernel(r2[1])) + (kernel(r2[2]) + kernel(r2[3]));
#pragma unroll 1
        for (int t = e + 1; t < 4; ++t) {
          const double wt = t == 2 ? w[2] : w[3];
#pragma unroll
          for (int s = 0; s < 4; ++s)
            c111 += kernel(fma(kGenA1, wt, r2[s])) + kernel(fma(-kGenA1, wt, r2[s]));
        }
      }
    }
#pragma unroll 1
    for (int m = 0; m < 4; ++m) {
      const double r1 = fma(m & 1 ? -kGenL : kGenL, w[0], fma(m & 2 ? -kGenL : kGenL, w[1], rc));
      const double rp = fma(kGenL, w[2], r1), rm = fma(-kGenL, w[2], r1);
      cl += (kernel(fma(kGenL, w[3], rp)) + kernel(fma(-kGenL, w[3], rp))) +
            (kernel(fma(kGenL, w[3], rm)) + kernel(fma(-kGenL, w[3], rm)));
    }

    // the groups together: (0) with (1, 2), then with (3 .. 6)
    const double e1 = fma(ea[0], b0, a0 * eb[0]), h1 = fma(ea[1], b0, a0 * eb[1]);
    const double e2 = fma(ea[0], eb[0], a0 * b11), e3 = ea[0] * b11;
    const double g = fma(ea[0], eb[1], fma(ea[1], eb[0], a0 * b12));
    out.S[0] = f0;
    out.S[1] = fma(e1, c0, ab * ec[0]);
    out.S[2] = fma(h1, c0, ab * ec[1]);
    out.S[3] = fma(fma(ea[2], b0, a0 * eb[2]), c0, ab * ec[2]);
    out.S[4] = fma(fma(ea[3], b0, a0 * eb[3]), c0, ab * ec[3]);
    out.S[5] = fma(e2, c0, fma(e1, ec[0], ab * c11));
    out.S[6] = fma(g, c0, fma(e1, ec[1], fma(h1, ec[0], ab * c12)));
    out.S[7] = fma(e3, c0, fma(e2, ec[0], fma(e1, c11, ab * c111)));
    out.S[8] = ea[4] * bl * cl;
    out.best = best;
    out.axis = axis;
  }
};

}  // namespace detail
}  // namespace cubature
