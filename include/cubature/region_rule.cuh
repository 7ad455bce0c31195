// region_rule.cuh -- the per-region degree-9 rule on the device.
//
// Computes, for one box [L, L+H], the five embedded rule sums, the
// fourth-difference split axis and the null-rule error estimate, i.e. what
// the reference does in SampleRegionBlock / computePermutation
// (quad/GPUquad/GPUQuadSample.cu:35-220), re-designed for sm_100a:
//
//  * K lanes (1..32, a power of two, inside one warp) cooperate on a region.
//    K = 1 is thread-per-region: every lane of a warp runs the same point
//    sequence on a different region, so control flow is uniform and no
//    cross-lane reduction is needed.  Small region lists use K = 8 or 32.
//  * Points are enumerated by generator structure, not decoded from a
//    permutation table: axes/axis pairs/triples come from a shared-memory
//    item table, signs are compile-time inner loops, and the coordinates of
//    a point are built with register selects from the region centre.  No
//    divergent __constant__ indexing, no per-point table reads.
//  * f is accumulated into one sum per generator set (the weights are
//    constant within a set); the five rule sums are formed once per region
//    (sum_k w[k][r] * S_k).  The Jacobian is applied once per region.
//  * Rule-sum finishing, null rules and the error heuristic use explicit
//    round-to-nearest intrinsics so they match the CPU oracle bit for bit
//    when the set sums agree.
#pragma once

#include <cstdint>

#include "rule9.hpp"

namespace cubature {
namespace detail {

// Axis combinations of the pair/triple generator sets, in the enumeration
// order the oracle uses (lexicographic; ordered pairs skip d2 == d1).
template <int N>
struct ItemTable {
  static constexpr int kPairs = N * (N - 1) / 2;
  static constexpr int kOPairs = N * (N - 1);
  static constexpr int kTriples = N * (N - 1) * (N - 2) / 6;
  uint32_t pair[kPairs > 0 ? kPairs : 1];
  uint32_t opair[kOPairs > 0 ? kOPairs : 1];
  uint32_t triple[kTriples > 0 ? kTriples : 1];

  // Filled by thread 0 of a block; callers synchronise afterwards.
  __device__ void fill() {
    int p = 0, o = 0, t = 0;
    for (int d1 = 0; d1 < N; ++d1)
      for (int d2 = d1 + 1; d2 < N; ++d2) pair[p++] = d1 | (d2 << 8);
    for (int d1 = 0; d1 < N; ++d1)
      for (int d2 = 0; d2 < N; ++d2)
        if (d2 != d1) opair[o++] = d1 | (d2 << 8);
    for (int d1 = 0; d1 < N; ++d1)
      for (int d2 = d1 + 1; d2 < N; ++d2)
        for (int d3 = d2 + 1; d3 < N; ++d3) triple[t++] = d1 | (d2 << 8) | (d3 << 16);
  }
};

// v[d] for a runtime d, as a select chain (keeps v in registers).
template <int N>
__device__ __forceinline__ double pick(const double (&v)[N], int d) {
  double r = v[0];
#pragma unroll
  for (int i = 1; i < N; ++i) r = (d == i) ? v[i] : r;
  return r;
}

// Per-region sums produced by the point loop (before the K-lane reduction).
struct RegionSums {
  double S[kNumSets];  // sum of f over each generator set
  double best;         // largest fourth difference seen
  int axis;            // its axis (smallest axis on ties)
};

// Coefficient of the box width for a coordinate with generator value +g
// (minus = false) or -g (minus = true): x = L + (0.5 - g) H.
__host__ __device__ __forceinline__ constexpr double coef(double g, bool minus) {
  return minus ? (0.5 + g) : (0.5 - g);
}

// Evaluate the point sums of one region for lane `lane` of K.  L and H are
// the box's lower corner and widths (global coordinates).
template <int N, int K, class F>
__device__ __forceinline__ void region_point_sums(const F& f, const double (&L)[N],
                                                  const double (&H)[N], int lane,
                                                  const ItemTable<N>& tab, double ratio,
                                                  RegionSums& out) {
#pragma unroll
  for (int k = 0; k < kNumSets; ++k) out.S[k] = 0;
  out.best = 0;
  out.axis = -1;

  double C[N];
#pragma unroll
  for (int i = 0; i < N; ++i) C[i] = fma(0.5, H[i], L[i]);

  // Set 0: the centre.  Every lane evaluates it (the fourth difference of
  // each axis needs it); lane 0 adds it.
  const double f0 = f(C);
  if (lane == 0) out.S[0] = f0;
  const double base = __dmul_rn(__dmul_rn(f0, 2.0), __dadd_rn(1.0, -ratio));

  // Sets 1-4: +-g on one axis.  Sets 1 and 2 give the fourth difference.
  for (int d = lane; d < N; d += K) {
    const double Ld = pick(L, d), Hd = pick(H, d);
    double fv[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const double g = (s < 2) ? kGenA1 : (s < 4) ? kGenA2 : (s < 6) ? kGenA3 : kGenA4;
      const double v = fma(coef(g, s & 1), Hd, Ld);
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = (i == d) ? v : C[i];
      fv[s] = f(x);
    }
    out.S[1] += fv[0];
    out.S[1] += fv[1];
    out.S[2] += fv[2];
    out.S[2] += fv[3];
    out.S[3] += fv[4];
    out.S[3] += fv[5];
    out.S[4] += fv[6];
    out.S[4] += fv[7];
    // |2(1-r) f0 + r (f1+ + f1-) - (f2+ + f2-)|  (GPUQuadSample.cu:155-162)
    const double fd = fabs(__dadd_rn(__dadd_rn(base, __dmul_rn(ratio, __dadd_rn(fv[0], fv[1]))),
                                     -__dadd_rn(fv[2], fv[3])));
    if (fd > out.best) {
      out.best = fd;
      out.axis = d;
    }
  }

  // Set 5: (+-a1, +-a1) on axis pairs d1 < d2.
  for (int t = lane; t < ItemTable<N>::kPairs; t += K) {
    const uint32_t it = tab.pair[t];
    const int d1 = it & 0xff, d2 = (it >> 8) & 0xff;
    const double L1 = pick(L, d1), H1 = pick(H, d1), L2 = pick(L, d2), H2 = pick(H, d2);
    const double v1p = fma(coef(kGenA1, false), H1, L1), v1m = fma(coef(kGenA1, true), H1, L1);
    const double v2p = fma(coef(kGenA1, false), H2, L2), v2m = fma(coef(kGenA1, true), H2, L2);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const double v1 = (s & 1) ? v1m : v1p, v2 = (s & 2) ? v2m : v2p;
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = (i == d1) ? v1 : ((i == d2) ? v2 : C[i]);
      out.S[5] += f(x);
    }
  }

  // Set 6: (+-a1 on d1, +-a2 on d2), ordered pairs d1 != d2.
  for (int t = lane; t < ItemTable<N>::kOPairs; t += K) {
    const uint32_t it = tab.opair[t];
    const int d1 = it & 0xff, d2 = (it >> 8) & 0xff;
    const double L1 = pick(L, d1), H1 = pick(H, d1), L2 = pick(L, d2), H2 = pick(H, d2);
    const double v1p = fma(coef(kGenA1, false), H1, L1), v1m = fma(coef(kGenA1, true), H1, L1);
    const double v2p = fma(coef(kGenA2, false), H2, L2), v2m = fma(coef(kGenA2, true), H2, L2);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const double v1 = (s & 1) ? v1m : v1p, v2 = (s & 2) ? v2m : v2p;
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = (i == d1) ? v1 : ((i == d2) ? v2 : C[i]);
      out.S[6] += f(x);
    }
  }

  // Set 7: (+-a1, +-a1, +-a1) on axis triples d1 < d2 < d3.
  for (int t = lane; t < ItemTable<N>::kTriples; t += K) {
    const uint32_t it = tab.triple[t];
    const int d1 = it & 0xff, d2 = (it >> 8) & 0xff, d3 = (it >> 16) & 0xff;
    const double L1 = pick(L, d1), H1 = pick(H, d1);
    const double L2 = pick(L, d2), H2 = pick(H, d2);
    const double L3 = pick(L, d3), H3 = pick(H, d3);
    const double v1p = fma(coef(kGenA1, false), H1, L1), v1m = fma(coef(kGenA1, true), H1, L1);
    const double v2p = fma(coef(kGenA1, false), H2, L2), v2m = fma(coef(kGenA1, true), H2, L2);
    const double v3p = fma(coef(kGenA1, false), H3, L3), v3m = fma(coef(kGenA1, true), H3, L3);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const double v1 = (s & 1) ? v1m : v1p, v2 = (s & 2) ? v2m : v2p, v3 = (s & 4) ? v3m : v3p;
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i)
        x[i] = (i == d1) ? v1 : ((i == d2) ? v2 : ((i == d3) ? v3 : C[i]));
      out.S[7] += f(x);
    }
  }

  // Set 8: (+-l, ..., +-l), all 2^N sign patterns; bit d of the pattern
  // makes coordinate d negative.  The low E bits run as a compile-time
  // inner loop, the high bits are one item.
  constexpr int E = N < 3 ? N : 3;
  constexpr int kItems8 = 1 << (N - E);
  double P[N], M[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    P[i] = fma(coef(kGenL, false), H[i], L[i]);
    M[i] = fma(coef(kGenL, true), H[i], L[i]);
  }
  for (int t = lane; t < kItems8; t += K) {
    double xh[N];
#pragma unroll
    for (int i = E; i < N; ++i) xh[i] = ((t >> (i - E)) & 1) ? M[i] : P[i];
#pragma unroll
    for (int s = 0; s < (1 << E); ++s) {
      double x[N];
#pragma unroll
      for (int i = 0; i < N; ++i) x[i] = (i < E) ? (((s >> i) & 1) ? M[i] : P[i]) : xh[i];
      out.S[8] += f(x);
    }
  }
}

// Functors whose value is a product over the axes (integrands.cuh).
template <class F, class = void>
struct AxisProductTrait {
  static constexpr bool value = false;
};
template <class F>
struct AxisProductTrait<F, decltype((void)F::kAxisProduct)> {
  static constexpr bool value = F::kAxisProduct;
};

// The rule's set sums over a product integrand as polynomials in the axes'
// factors (axis_product_sums), over some of the axes: z centres only; e1,
// e2, e3 one, two, three axes at a1; h1 one axis at a2; g one axis at a1 and
// one at a2; p, q one axis at a3, a4; l corners.
struct AxisPoly {
  double z = 1, e1 = 0, e2 = 0, e3 = 0, h1 = 0, g = 0, p = 0, q = 0, l = 1;

  // Append one axis with centre factor c and factor sums s, w, tp, tq, tl.
  __device__ __forceinline__ void append(double c, double s, double w, double tp, double tq,
                                         double tl) {
    e3 = fma(e3, c, e2 * s);
    e2 = fma(e2, c, e1 * s);
    g = fma(g, c, fma(e1, w, h1 * s));
    e1 = fma(e1, c, z * s);
    h1 = fma(h1, c, z * w);
    p = fma(p, c, z * tp);
    q = fma(q, c, z * tq);
    l *= tl;
    z *= c;
  }

  // Those of two disjoint groups of axes together.
  __device__ __forceinline__ static AxisPoly join(const AxisPoly& a, const AxisPoly& b) {
    AxisPoly r;
    r.e3 = fma(a.e3, b.z, fma(a.e2, b.e1, fma(a.e1, b.e2, a.z * b.e3)));
    r.e2 = fma(a.e2, b.z, fma(a.e1, b.e1, a.z * b.e2));
    r.g = fma(a.g, b.z, fma(a.e1, b.h1, fma(a.h1, b.e1, a.z * b.g)));
    r.e1 = fma(a.e1, b.z, a.z * b.e1);
    r.h1 = fma(a.h1, b.z, a.z * b.h1);
    r.p = fma(a.p, b.z, a.z * b.p);
    r.q = fma(a.q, b.z, a.z * b.q);
    r.l = a.l * b.l;
    r.z = a.z * b.z;
    return r;
  }

  // This and the polynomials of the lane `off` above in the K-lane group
  // (complete in lane 0 after off = 1, 2, ..., K / 2).
  template <int K>
  __device__ __forceinline__ void join_down(unsigned mask, int off) {
    AxisPoly o;
    o.z = __shfl_down_sync(mask, z, off, K);
    o.e1 = __shfl_down_sync(mask, e1, off, K);
    o.e2 = __shfl_down_sync(mask, e2, off, K);
    o.e3 = __shfl_down_sync(mask, e3, off, K);
    o.h1 = __shfl_down_sync(mask, h1, off, K);
    o.g = __shfl_down_sync(mask, g, off, K);
    o.p = __shfl_down_sync(mask, p, off, K);
    o.q = __shfl_down_sync(mask, q, off, K);
    o.l = __shfl_down_sync(mask, l, off, K);
    *this = join(*this, o);
  }

  __device__ __forceinline__ void store(RegionSums& out) const {
    out.S[0] = z;
    out.S[1] = e1;
    out.S[2] = h1;
    out.S[3] = p;
    out.S[4] = q;
    out.S[5] = e2;
    out.S[6] = g;
    out.S[7] = e3;
    out.S[8] = l;
  }
};

// The split axis of a product integrand: the axis of the largest fourth
// difference |2 (1 - r) f0 + r (f1+ + f1-) - (f2+ + f2-)| (set-1 and set-2
// values), the smallest such axis on ties, -1 when all are zero.
//
// Axis d's difference over f0 is |2 (1 - r) + (r s - w) / c|, from the
// factors at hand.  It decides when the largest leaves the second behind by
// more than both ways of computing it can be off; else (ties of symmetric
// integrands, differences down in the rounding) exact_axis evaluates the
// points one by one with the fold of operator(), the same bits as f(x), and
// compares those as the point-by-point evaluators do.
struct AxisChoice {
  double best = 0, second = 0, scale = 0;
  int axis = -1;

  // Axis d: centre factor c >= 0 and factor sums s, w at a1, a2, all of them
  // times inv (> 0) over f0.
  __device__ __forceinline__ void add(int d, double inv, double c, double s, double w,
                                      double ratio) {
    const double k = 2.0 * (1.0 - ratio);
    const double v = fabs(fma(k, c, fma(ratio, s, -w))) * inv;
    scale = fmax(scale, fma(k, c, fma(ratio, fabs(s), fabs(w))) * inv);
    if (v > best) {
      second = best;
      best = v;
      axis = d;
    } else {
      second = v <= second ? second : v;  // NaN stays
    }
  }

  template <int K>
  __device__ __forceinline__ void join_lanes(unsigned mask, int off) {
    join(__shfl_xor_sync(mask, best, off, K), __shfl_xor_sync(mask, second, off, K),
         __shfl_xor_sync(mask, axis, off, K), __shfl_xor_sync(mask, scale, off, K));
  }
  template <int K>
  __device__ __forceinline__ void join_down(unsigned mask, int off) {
    join(__shfl_down_sync(mask, best, off, K), __shfl_down_sync(mask, second, off, K),
         __shfl_down_sync(mask, axis, off, K), __shfl_down_sync(mask, scale, off, K));
  }
  __device__ __forceinline__ void join(double ob, double os, int oa, double oscale) {
    scale = fmax(scale, oscale);
    const double m = second <= os ? os : second, lo = ob <= best ? ob : best;
    second = m <= lo ? lo : m;
    if (ob > best) {
      best = ob;
      axis = oa;
    }
  }

  // f0: the product of the centre factors (too small a value may be zero as
  // the fold forms it)
  __device__ __forceinline__ bool sure(double noise, double f0) const {
    return best - second > noise * scale && scale < 1e290 && f0 > 1e-280;
  }
};

template <int N, class F, class V, class Box>
__device__ __noinline__ int exact_axis(const V& f, const Box& box, double ratio) {
  double tc[N];
  double acc = F::start();
#pragma unroll 1
  for (int i = 0; i < N; ++i) {
    tc[i] = f.axis(i).term(fma(0.5, box.len(i), box.lo(i)));
    acc = F::step(acc, tc[i]);
  }
  const double f0 = F::finish(acc);
  const double base = __dmul_rn(__dmul_rn(f0, 2.0), __dadd_rn(1.0, -ratio));
  double pre = F::start(), best = 0;
  int axis = -1;
#pragma unroll 1
  for (int d = 0; d < N; ++d) {
    const auto ax = f.axis(d);
    const double Ld = box.lo(d), Hd = box.len(d);
    double v[4];
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      const double c = k == 0   ? coef(kGenA1, false)
                       : k == 1 ? coef(kGenA1, true)
                       : k == 2 ? coef(kGenA2, false)
                                : coef(kGenA2, true);
      double t = F::step(pre, ax.term(fma(c, Hd, Ld)));
      for (int i = d + 1; i < N; ++i) t = F::step(t, tc[i]);
      v[k] = F::finish(t);
    }
    const double fd = fabs(__dadd_rn(__dadd_rn(base, __dmul_rn(ratio, __dadd_rn(v[0], v[1]))),
                                     -__dadd_rn(v[2], v[3])));
    if (fd > best) {
      best = fd;
      axis = d;
    }
    pre = F::step(pre, tc[d]);
  }
  return axis;
}

// The same choice from the values of the points themselves, for any functor:
// the comparisons of region_point_sums, with the bits of f(x).
template <int N, class F>
__device__ __noinline__ int exact_axis_points(const F& f, const double (&L)[N],
                                              const double (&H)[N], double ratio) {
  double x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = fma(0.5, H[i], L[i]);
  const double base = __dmul_rn(__dmul_rn(f(x), 2.0), __dadd_rn(1.0, -ratio));
  double best = 0;
  int axis = -1;
#pragma unroll 1
  for (int d = 0; d < N; ++d) {
    const double c = x[d];
    double v[4];
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      const double g = k == 0   ? coef(kGenA1, false)
                       : k == 1 ? coef(kGenA1, true)
                       : k == 2 ? coef(kGenA2, false)
                                : coef(kGenA2, true);
      x[d] = fma(g, H[d], L[d]);
      v[k] = f(x);
    }
    x[d] = c;
    const double fd = fabs(__dadd_rn(__dadd_rn(base, __dmul_rn(ratio, __dadd_rn(v[0], v[1]))),
                                     -__dadd_rn(v[2], v[3])));
    if (fd > best) {
      best = fd;
      axis = d;
    }
  }
  return axis;
}

// Set sums and fourth difference of one region by one thread, for
// integrands that are products over the axes (AxisProductTrait).
//
// With centre factors c_i and, per axis, the sums of the factors at +-g for
// each generator g (s: a1, w: a2, p: a3, q: a4, l: corner), the distributive
// law turns each set's sum over its 2N ... 2^N points into a polynomial in
// these: sets 3 and 4 are sum_i p_i prod_{j != i} c_j, set 5 the sum over
// pairs s_i s_j, set 6 over ordered pairs s_i w_j, set 7 over triples
// s_i s_j s_k (each times the other axes' centres), set 8 prod l_i.  One
// pass over the axes builds all of them by appending an axis at a time.
// Every quantity is a sum of products of like sign where the factors are
// positive, so nothing cancels.
//
// About 1 k FP64 instructions for a 6-D product peak instead of 13.6 k point
// by point (453 points): the per-step rule over 1 M 6-D regions went from 1197
// to 93 us (product peak) and from 1895 to 195 us (Gaussian) on a B200, bound
// by FP64 issue.  The loop over the axes stays rolled: ten
// independent terms per axis are parallelism enough, and unrolled over the
// axes the Gaussian's exponentials spilled 2.5 KB a thread.  The box is read
// per axis (box.lo(d), box.len(d)) instead of being held in registers, which
// a rolled loop cannot index.
//
// V: the functor, or a view of its parameters (axis(i)); F: the functor's
// type.  jac receives the box volume.
template <class F, class V, class Box>
__device__ __forceinline__ void append_axis(const V& f, const Box& box, int d, double ratio,
                                            AxisPoly& poly, AxisChoice& ch, double& vol) {
  const auto ax = f.axis(d);
  const double Ld = box.lo(d), Hd = box.len(d);
  auto at = [&](double gen, bool minus) { return ax.term(fma(coef(gen, minus), Hd, Ld)); };
  const double tc = ax.term(fma(0.5, Hd, Ld)), c = F::factor(tc);
  const double s = F::factor2(at(kGenA1, false), at(kGenA1, true));
  const double w = F::factor2(at(kGenA2, false), at(kGenA2, true));
  ch.add(d, F::inverse(tc, c), c, s, w, ratio);
  poly.append(c, s, w, F::factor2(at(kGenA3, false), at(kGenA3, true)),
              F::factor2(at(kGenA4, false), at(kGenA4, true)),
              F::factor2(at(kGenL, false), at(kGenL, true)));
  vol = __dmul_rn(vol, Hd);
}

// Lanes to an axis with K lanes to a region: with 16, what the axes leave room
// for, up to one for each of the five sums.
constexpr int split_share(int n, int k) { return k < 16 ? 1 : k / n < 5 ? k / n : 5; }

// append_axis of axis j / R by R lanes (j: lane in the K-lane group): the five
// sums are dealt to them, and every lane appends all of the axis.
template <int N, int K, int R, class F, class V, class Box>
__device__ __forceinline__ void append_axis_lanes(const V& f, const Box& box, int j, unsigned mask,
                                                  double ratio, AxisPoly& poly, AxisChoice& ch,
                                                  double& vol) {
  constexpr int kRounds = (5 + R - 1) / R;
  const int d = j / R, first = d < N ? d * R : 0;
  double tc = 0, c = 0, len = 0, v[kRounds];
#pragma unroll
  for (int a = 0; a < kRounds; ++a) v[a] = 0;
  if (d < N) {
    const auto ax = f.axis(d);
    const double Ld = box.lo(d);
    len = box.len(d);
    tc = ax.term(fma(0.5, len, Ld));
    c = F::factor(tc);
#pragma unroll
    for (int a = 0; a < kRounds; ++a) {
      const int item = j - first + a * R;
      const double g = item == 0   ? kGenA1
                       : item == 1 ? kGenA2
                       : item == 2 ? kGenA3
                       : item == 3 ? kGenA4
                                   : kGenL;
      if (item < 5)
        v[a] = F::factor2(ax.term(fma(coef(g, false), len, Ld)),
                          ax.term(fma(coef(g, true), len, Ld)));
    }
  }
  __syncwarp(mask);
  double all[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) all[i] = __shfl_sync(mask, v[i / R], first + i % R, K);
  if (d < N) {
    ch.add(d, F::inverse(tc, c), c, all[0], all[1], ratio);
    poly.append(c, all[0], all[1], all[2], all[3], all[4]);
    vol = __dmul_rn(vol, len);
  }
}

template <int N, class F, class V, class Box>
__device__ __forceinline__ void axis_product_sums(const V& f, const Box& box, double ratio,
                                                  RegionSums& out, double& jac) {
  AxisPoly poly;
  AxisChoice ch;
  jac = 1;
#pragma unroll 1
  for (int d = 0; d < N; ++d) append_axis<F>(f, box, d, ratio, poly, ch, jac);
  poly.store(out);
  out.best = ch.best;
  out.axis = ch.sure(F::noise(poly.z), poly.z) ? ch.axis : exact_axis<N, F>(f, box, ratio);
}

// axis_product_sums with the axes dealt to the K lanes of a group (lane j: a
// run of neighbouring axes), for chains of dependent regions, where the
// latency of one region counts: a lane evaluates its axes' factors, and the
// lanes' polynomials are joined by shuffles.  Every lane of the group (mask, K
// aligned lanes) gets the sums.
//
// The sums have the same bits for every K that gives a lane one axis or two:
// appending an axis to another is joining the two (the terms that append
// leaves out are products with zeros), and lanes of two axes start with the
// pairs that lanes of one axis join first.  So a box is refined the same way
// whichever K its call takes.  (With axes j and j + K on lane j the last bits
// changed with K.)  With several lanes to an axis (K = 16) the lanes of an axis
// share its factors, and the joins are those of a lane per axis.
template <int N, int K, class F, class V, class Box>
__device__ __forceinline__ void axis_split_sums(const V& f, const Box& box, int j, unsigned mask,
                                                double ratio, RegionSums& out, double& jac) {
  AxisPoly poly;
  AxisChoice ch;
  jac = 1;
  constexpr int kPer = (N + K - 1) / K;
  static_assert(kPer <= 2, "the joins' order depends on K");
  constexpr int kShare = split_share(N, K);
  if constexpr (kShare > 1) {
    append_axis_lanes<N, K, kShare, F>(f, box, j, mask, ratio, poly, ch, jac);
#pragma unroll
    for (int off = kShare; off < N * kShare; off <<= 1) {
      poly.template join_down<K>(mask, off);
      ch.template join_down<K>(mask, off);
      jac = __dmul_rn(jac, __shfl_down_sync(mask, jac, off, K));
    }
    // complete in lane 0
    poly.store(out);
    out.best = ch.best;
    out.axis = ch.sure(F::noise(poly.z), poly.z) ? ch.axis : -2;
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) out.S[k] = __shfl_sync(mask, out.S[k], 0, K);
    jac = __shfl_sync(mask, jac, 0, K);
    out.axis = __shfl_sync(mask, out.axis, 0, K);
    if (out.axis == -2) out.axis = exact_axis<N, F>(f, box, ratio);
  } else {
    const int d1 = (j + 1) * kPer < N ? (j + 1) * kPer : N;
#pragma unroll 1
    for (int d = j * kPer; d < d1; ++d) append_axis<F>(f, box, d, ratio, poly, ch, jac);
    __syncwarp(mask);
#pragma unroll
    for (int off = 1; off < K; off <<= 1) {
      poly.template join_down<K>(mask, off);
      ch.template join_lanes<K>(mask, off);
      jac = __dmul_rn(jac, __shfl_xor_sync(mask, jac, off));
    }
    poly.store(out);
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) out.S[k] = __shfl_sync(mask, out.S[k], 0, K);
    out.best = ch.best;
    out.axis = ch.sure(F::noise(out.S[0]), out.S[0]) ? ch.axis : exact_axis<N, F>(f, box, ratio);
  }
}

// A box in an SoA region list.
struct ListBox {
  const double* lo0;
  const double* len0;
  long long ld;
  __device__ __forceinline__ double lo(int d) const { return lo0[d * ld]; }
  __device__ __forceinline__ double len(int d) const { return len0[d * ld]; }
};

// Functors with an evaluator of their own for one region by one thread:
// ThreadSums<F>::run(f, L, H, ratio, out).  kMinList: the list length from
// which it beats several lanes per region.
template <class F>
struct ThreadSums {
  static constexpr bool value = false;
  static constexpr int kMinList = 0;
};

// One thread per region has a form that shares work between the rule's
// points: it is then the faster one for every list length, or from kMinList
// on; else only for lists that fill the chip.
template <class F>
constexpr bool kFactored = AxisProductTrait<F>::value || ThreadSums<F>::value;

// The sums of one region of a factored integrand by one thread, and its
// volume.
template <int N, class F, class V, class Box>
__device__ __forceinline__ void factored_sums(const V& f, const Box& box, double ratio,
                                              RegionSums& out, double& jac) {
  if constexpr (AxisProductTrait<F>::value) {
    axis_product_sums<N, F>(f, box, ratio, out, jac);
  } else {
    double L[N], H[N];
    jac = 1;
#pragma unroll
    for (int d = 0; d < N; ++d) {
      L[d] = box.lo(d);
      H[d] = box.len(d);
      jac = __dmul_rn(jac, H[d]);
    }
    ThreadSums<F>::run(f, L, H, ratio, out);
  }
}

// The sums of one region by one thread, and its volume.
template <int N, class F, class V, class Box>
__device__ __forceinline__ void thread_sums(const V& f, const Box& box, const ItemTable<N>& tab,
                                            double ratio, RegionSums& out, double& jac) {
  if constexpr (kFactored<F>) {
    factored_sums<N, F>(f, box, ratio, out, jac);
  } else {
    double L[N], H[N];
    jac = 1;
#pragma unroll
    for (int d = 0; d < N; ++d) {
      L[d] = box.lo(d);
      H[d] = box.len(d);
      jac = __dmul_rn(jac, H[d]);
    }
    region_point_sums<N, 1>(f, L, H, 0, tab, ratio, out);
  }
}

// Combine the sums of the K lanes of a group (xor butterfly inside the
// aligned K-lane group).  Ties of the fourth difference keep the smaller
// axis, as the reference's strict '>' scan does.
template <int K>
__device__ __forceinline__ void reduce_lanes(RegionSums& r, unsigned mask) {
#pragma unroll
  for (int off = K / 2; off > 0; off >>= 1) {
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) r.S[k] += __shfl_xor_sync(mask, r.S[k], off);
    const double ob = __shfl_xor_sync(mask, r.best, off);
    const int oa = __shfl_xor_sync(mask, r.axis, off);
    const bool take = (ob > r.best) || (ob == r.best && oa >= 0 && (r.axis < 0 || oa < r.axis));
    if (take) {
      r.best = ob;
      r.axis = oa;
    }
  }
}

struct RegionResult {
  double avg, err;
  int axis;
};

// Rule sums -> value, null-rule error, split axis (GPUQuadSample.cu:195-216).
// jac is the box volume times 2^-div; fallback_axis is used when every
// fourth difference is zero.
template <int N>
__device__ __forceinline__ RegionResult finish_region(const RegionSums& r, const RuleTables& T,
                                                      double jac, int fallback_axis) {
  double sum[kNumRules];
#pragma unroll
  for (int q = 0; q < kNumRules; ++q) {
    double acc = 0;
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) acc = __dadd_rn(acc, __dmul_rn(T.wt[k][q], r.S[k]));
    sum[q] = __dmul_rn(acc, jac);
  }
  double nul[kNumRules];
#pragma unroll
  for (int q = 1; q < kNumRules - 1; ++q) {
    double m = 0;
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) {
      const double e =
          __dmul_rn(fabs(__dadd_rn(sum[q + 1], __dmul_rn(T.scale[k][q], sum[q]))), T.norm[k][q]);
      m = (m > e) ? m : e;
    }
    nul[q] = m;
  }
  RegionResult out;
  out.avg = sum[0];
  const double m12 = nul[1] > nul[2] ? nul[1] : nul[2];
  const double m123 = m12 > nul[3] ? m12 : nul[3];
  out.err = (__dmul_rn(5.0, nul[1]) <= nul[2] && __dmul_rn(5.0, nul[2]) <= nul[3])
                ? nul[1]
                : __dmul_rn(5.0, m123);
  out.axis = r.axis >= 0 ? r.axis : fallback_axis;
  return out;
}

// finish_region with the rules dealt to the K lanes of a group, each with
// finish_region's arithmetic for its rule.  T is read by lane index, so it
// must lie in shared memory.  Every lane gets the result.
template <int K>
__device__ __forceinline__ RegionResult finish_region_split(const RegionSums& r,
                                                            const RuleTables& T, double jac,
                                                            int fallback_axis, int j,
                                                            unsigned mask) {
  double sum[kNumRules];
#pragma unroll
  for (int a = 0; a < (kNumRules + K - 1) / K; ++a) {
    const int q = j + a * K < kNumRules ? j + a * K : 0;
    double acc = 0;
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) acc = __dadd_rn(acc, __dmul_rn(T.wt[k][q], r.S[k]));
    acc = __dmul_rn(acc, jac);
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (a * K + i < kNumRules) sum[a * K + i] = __shfl_sync(mask, acc, i, K);
  }
  double nul[kNumRules];
#pragma unroll
  for (int a = 0; a < (kNumRules - 2 + K - 1) / K; ++a) {
    const int q = 1 + (j + a * K < kNumRules - 2 ? j + a * K : 0);
    const double sq = q == 1 ? sum[1] : q == 2 ? sum[2] : sum[3];
    const double sq1 = q == 1 ? sum[2] : q == 2 ? sum[3] : sum[4];
    double m = 0;
#pragma unroll
    for (int k = 0; k < kNumSets; ++k) {
      const double e = __dmul_rn(fabs(__dadd_rn(sq1, __dmul_rn(T.scale[k][q], sq))), T.norm[k][q]);
      m = (m > e) ? m : e;
    }
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (a * K + i < kNumRules - 2) nul[1 + a * K + i] = __shfl_sync(mask, m, i, K);
  }
  RegionResult out;
  out.avg = sum[0];
  const double m12 = nul[1] > nul[2] ? nul[1] : nul[2];
  const double m123 = m12 > nul[3] ? m12 : nul[3];
  out.err = (__dmul_rn(5.0, nul[1]) <= nul[2] && __dmul_rn(5.0, nul[2]) <= nul[3])
                ? nul[1]
                : __dmul_rn(5.0, m123);
  out.axis = r.axis >= 0 ? r.axis : fallback_axis;
  return out;
}

}  // namespace detail
}  // namespace cubature
