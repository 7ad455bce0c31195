// step_kernels.cuh -- stand-alone kernels behind the per-step C entry points
// (rule evaluation, split, reduction on caller-provided buffers).  The
// engine fuses the same work into its own iteration kernels.
#pragma once

#include "engine_kernels.cuh"

namespace cubature {

// List length from which k_step_rule takes one thread per region (below: a
// warp).  Point by point: when the list fills the chip.
template <class F>
inline long long rule_thread_min(int sms) {
  return detail::kFactored<F> ? detail::ThreadSums<F>::kMinList : sms * 512ll;
}

// Rule + classification over one integral's SoA list (INTEGRATE_GPU_PHASE1,
// GPUQuadPhases.cu:38-79).
template <int N, int K, class F>
__global__ void __launch_bounds__((K == 1 && detail::kFactored<F>) ? 128 : 256) k_step_rule(F f, RuleTables T, long long n,
                                                   const double* lo, const double* len,
                                                   long long ld, double epsrel, double epsabs,
                                                   double* avg, double* err, int* axis,
                                                   int* active) {
  __shared__ detail::ItemTable<N> tab;
  if (threadIdx.x == 0) tab.fill();
  __syncthreads();
  const int kGroups = (int)blockDim.x / K;
  const int lane = threadIdx.x % K;
  const unsigned gmask =
      (K == 32) ? 0xffffffffu : (((1u << K) - 1u) << ((threadIdx.x & 31) & ~(K - 1)));
  for (long long i = (long long)blockIdx.x * kGroups + threadIdx.x / K; i < n;
       i += (long long)gridDim.x * kGroups) {
    detail::RegionSums rs;
    double jac;
    if constexpr (K == 1) {
      detail::thread_sums<N, F>(f, detail::ListBox{lo + i, len + i, ld}, tab, T.ratio, rs, jac);
    } else {
      double L[N], H[N];
#pragma unroll
      for (int d = 0; d < N; ++d) {
        L[d] = lo[(long long)d * ld + i];
        H[d] = len[(long long)d * ld + i];
      }
      detail::region_point_sums<N, K>(f, L, H, lane, tab, T.ratio, rs);
      detail::reduce_lanes<K>(rs, gmask);
      jac = 1;
#pragma unroll
      for (int d = 0; d < N; ++d) jac = __dmul_rn(jac, H[d]);
    }
    if (lane == 0) {
      const detail::RegionResult r = detail::finish_region<N>(rs, T, jac, 0);
      avg[i] = r.avg;
      err[i] = r.err;
      axis[i] = r.axis;
      active[i] = (r.err / detail::max_err(r.avg, epsrel, epsabs)) > 1;
    }
  }
}

// Split, pass 1: active count per 32-region chunk.
static __global__ void k_step_count(long long n, const int* active, int* cnt) {
  const int lane = threadIdx.x & 31;
  const long long nchunk = (n + 31) / 32;
  for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32; c < nchunk;
       c += (long long)gridDim.x * blockDim.x / 32) {
    const long long i = c * 32 + lane;
    const unsigned b = __ballot_sync(0xffffffffu, i < n && active[i] == 1);
    if (lane == 0) cnt[c] = __popc(b);
  }
}

// Split, pass 2: exclusive scan of the chunk counts (one block, 16 chunks a
// thread and pass); writes the child count 2m.  One chunk a thread took 33 us
// for the 31 k chunks of 1 M regions, a block-wide scan and its barriers per
// 1024 of them.
constexpr int kScanPer = 16;
static __global__ void __launch_bounds__(1024) k_step_scan(long long nchunk, const int* cnt, int* excl,
                                                    long long* count_out) {
  __shared__ long long wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  long long carry = 0;
  for (long long base = 0; base < nchunk; base += 1024 * kScanPer) {
    const long long c0 = base + (long long)tid * kScanPer;
    int v[kScanPer];
    long long sum = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
      v[i] = c0 + i < nchunk ? cnt[c0 + i] : 0;
      sum += v[i];
    }
    long long incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    long long w = wsum[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += t;
    }
    const long long before = __shfl_sync(0xffffffffu, w, wid > 0 ? wid - 1 : 0);
    long long run = carry + (wid > 0 ? before : 0) + incl - sum;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
      if (c0 + i < nchunk) excl[c0 + i] = (int)run;
      run += v[i];
    }
    carry += __shfl_sync(0xffffffffu, w, 31);
    __syncthreads();  // wsum is read before the next pass writes it
  }
  if (tid == 0) *count_out = 2 * carry;
}

// Split, pass 3: write the children (alignRegions + divideIntervalsGPU,
// GPUKernelquad.cu:63-149).
template <int N>
__global__ void k_step_write(long long n, const double* lo, const double* len, long long ld,
                             const int* active, const int* axis, const int* excl,
                             const long long* count, double* olo, double* olen, long long old,
                             int layout) {
  const int lane = threadIdx.x & 31;
  const long long nchunk = (n + 31) / 32;
  const long long m = *count / 2;
  for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32; c < nchunk;
       c += (long long)gridDim.x * blockDim.x / 32) {
    const long long i = c * 32 + lane;
    const bool act = i < n && active[i] == 1;
    const unsigned b = __ballot_sync(0xffffffffu, act);
    if (!act) continue;
    const long long j = excl[c] + __popc(b & ((1u << lane) - 1u));
    const long long d0 = layout == 0 ? j : 2 * j;
    const long long d1 = layout == 0 ? m + j : 2 * j + 1;
    const int ax = axis[i];
#pragma unroll
    for (int d = 0; d < N; ++d) {
      const double l = lo[(long long)d * ld + i], w = len[(long long)d * ld + i];
      const double h = w / 2;
      olo[(long long)d * old + d0] = l;
      olo[(long long)d * old + d1] = d == ax ? l + 1 * h : l;
      olen[(long long)d * old + d0] = d == ax ? h : w;
      olen[(long long)d * old + d1] = d == ax ? h : w;
    }
  }
}

// Reduction, pass 1: per-block partial sums (fixed grid, fixed order).
constexpr int kReduceBlocks = 1024;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

static __global__ void __launch_bounds__(256) k_step_reduce(long long n, const double* avg,
                                                     const double* err, const int* active,
                                                     double* part) {
  __shared__ double sm[8][4];
  double s[4] = {0, 0, 0, 0};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const double a = avg[i], e = err[i];
    s[0] += a;
    s[1] += e;
    if (active[i] != 1) {
      s[2] += a;
      s[3] += e;
    }
  }
  for (int q = 0; q < 4; ++q) s[q] = warp_sum(s[q]);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
    for (int q = 0; q < 4; ++q) sm[wid][q] = s[q];
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0;
    for (int w = 0; w < 8; ++w) t += sm[w][threadIdx.x];
    part[blockIdx.x * 4 + threadIdx.x] = t;
  }
}

// Reduction, pass 2: a warp per sum, lane-strided over the block partials in a
// fixed order (one warp for all four read 128 bytes a step and took 10 us).
static __global__ void __launch_bounds__(128) k_step_reduce_final(int nblocks, const double* part,
                                                                  double* out) {
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  double s = 0;
#pragma unroll 8
  for (int b = lane; b < nblocks; b += 32) s += part[b * 4 + q];
  s = warp_sum(s);
  if (lane == 0) out[q] = s;
}

}  // namespace cubature
