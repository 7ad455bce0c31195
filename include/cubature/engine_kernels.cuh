// engine_kernels.cuh -- the device side of the breadth-first engine.
//
// One iteration of the reference's first phase (GPUKernelquad.cu:509-605)
// over a batch of independent integrals whose regions share one list:
//
//   eval      rule + fourth difference + error + classification per region
//             (INTEGRATE_GPU_PHASE1, GPUQuadPhases.cu:38-79)
//   partials  per 32-region chunk: value/error sums, finished sums, active
//             count (the reference's four thrust::reduce calls and the
//             exclusive scan, GPUKernelquad.cu:364-386,565-577)
//   decide    per integral: totals, the global stop test, the child count
//             (GPUKernelquad.cu:583-598)
//   scan      exclusive scan of child counts over integrals -> new segments
//   split     compaction + bisection of the active regions, written as
//             adjacent children (alignRegions + divideIntervalsGPU,
//             GPUKernelquad.cu:63-149)
//
// The steps are warp-level device functions shared by two drivers: one
// kernel launch per step (the throughput regime, engine.cuh) and the
// persistent cooperative kernel (the latency regime, persistent.cuh).
//
// Layout in HBM: region lists are SoA, lo[d * cap + i] and len[d * cap + i]
// (FP64), rid[i] = owning integral (-1 = padding).  Each integral owns a
// contiguous segment whose start is a multiple of 32, so a 32-region chunk
// never straddles two integrals and every reduction is a fixed-order tree
// (results are bit-reproducible run to run).
#pragma once

#include <cstdint>
#include <type_traits>
#include <utility>

#include "integrands.cuh"
#include "linear_sums.cuh"
#include "region_rule.cuh"

namespace cubature {

enum Policy : int { kPolicyReference = 0, kPolicyBreadth = 1 };

// Status of an integral whose sums stopped being finite (a NaN or infinite
// integrand value), CUB_STATUS_NONFINITE of the C ABI.
constexpr int kStatusNonFinite = 1 << 30;

enum IntegralStateCode : int {
  kStateRunning = 0,
  kStateDone = 1,      // converged or out of active regions
  kStatePhase2 = 2,    // handed to the depth-first second phase
  kStateCapacity = 3,  // stopped: region capacity or iteration limit
};

// Per-integral state, resident on the device for the whole run.
struct IntegralState {
  double epsrel, epsabs;
  double value, error;  // finished sums (final results when done)
  double last_value, last_error;
  unsigned long long nregions, neval;
  int state, status, iters;
  int left_new;                // leftover boxes produced this iteration
  int seg_start, seg_count;    // segment in the current list
  int next_start, next_count;  // segment in the next list
  int left_start, left_count;  // leftover boxes for phase 2
  // persistent kernel, where the next list is built lazily: the segment
  // of the list the current one was split from, and the global iteration
  // whose first step copies this integral's leftovers (hand-off to phase 2)
  int par_start, par_count;
  int handoff_at, pad;
};

struct ChunkPartial {
  double sum_avg, sum_err;  // all regions of the chunk
  double fin_avg, fin_err;  // finished regions only
  int nactive;
  unsigned mask;  // bit i: slot 32c + i stays active
};

// Sums of kTileChunks consecutive chunks of one integral (its chunks
// kTileChunks t .. kTileChunks t + kTileChunks - 1, counted from the
// start of its segment).
constexpr int kTileChunks = 256;
struct TileSum {
  double sum_avg, sum_err, fin_avg, fin_err;
  int nactive;
  int base;  // active regions of the integral before the tile
};

// List sizes after one iteration's scan.
struct IterState {
  int n;          // slots in the list (padded)
  int n_running;  // integrals with regions in that list
  int n_left;     // leftover boxes queued for phase 2 so far
  int overflow;   // the list or the leftovers would exceed capacity
  int handoff;    // some integral was handed to phase 2 by this scan
};

// Control block shared by the host and both drivers.
struct Control {
  IterState host;      // result of the last scan (multi-launch driver)
  IterState it[2];     // double-buffered by iteration parity (persistent)
  int cur;             // index of the current list buffer
  int iters_done;      // breadth-first iterations completed
  int exit_reason;     // persistent kernel: why it returned
  int pad;
  unsigned done_cnt;   // integrals decided in this iteration
  unsigned bar_count;  // grid barrier arrivals since the launch (monotonic)
  unsigned exit_count;  // replicated kernel: blocks that have left this launch
  int timeout;         // a bounded wait gave up
  // globaltimer stamps (ns) of the persistent kernels' first kTraceIters
  // iterations, kTraceSlots per iteration (diagnostics, read back with the
  // control block).  Persistent kernel: 0 start, 1 next list assigned,
  // 2 grid barrier passed, 3 decider read its integral state, 4 block 0's
  // evaluations done, 5 last chunk summed, 6 integrals decided, 7 chunk sums
  // combined.  Replicated kernel (block 0): 0 start, 7 first region set up,
  // 4 evaluations done, 2 grid barrier passed, 3 chunk partials formed,
  // 1 per-integral sums formed (warp 0), 6 stop decision taken, 5 next
  // segments assigned.
  unsigned long long trace[64];
};
constexpr int kTraceIters = 8;
constexpr int kTraceSlots = 8;

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void trace_mark(Control* ctl, int it, int slot) {
  if (it < kTraceIters) ctl->trace[kTraceSlots * it + slot] = global_ns();
}

enum ExitReason : int {
  kExitDone = 1,      // no integral left running
  kExitLarge = 2,     // the list grew past the persistent kernel's range
  kExitCapacity = 3,  // buffers must grow before the next iteration
  kExitTimeout = 4,   // a grid barrier wait ran out
};

struct EngineArgs {
  // current list
  const double* lo;
  const double* len;
  const int* rid;
  int n;  // padded slot count
  long long cap;
  // per-region outputs
  double* avg;
  double* err;
  int* axis;
  int* active;
  // chunk partials / prefix / arrival counters
  ChunkPartial* part;
  int* chunk_excl;
  TileSum* tile;    // multi-launch driver: sums of whole tiles; else null
  unsigned* cmask;  // active bit mask per chunk (optional)
  unsigned* chunk_cnt;
  unsigned* int_cnt;
  // next list
  double* nlo;
  double* nlen;
  int* nrid;
  long long ncap;
  // leftovers for phase 2
  double* left_lo;
  double* left_len;
  int* left_rid;
  long long left_cap;
  // integrals
  IntegralState* ist;
  int nint;
  Control* ctl;
  int policy;
  int phase1_cap;  // child count that ends phase 1 (0 = never)
  int max_iters;   // phase-1 iteration limit
  int npoints;
};

namespace detail {

__host__ __device__ __forceinline__ double max_err(double avg, double epsrel, double epsabs) {
  const double a = epsrel * fabs(avg);
  return a > epsabs ? a : epsabs;
}

template <class F>
struct SingleSource {
  F f;
  __device__ __forceinline__ const F& get(int) const { return f; }
};

// Functor F's axis parameters read from a parameter block as they are used.
template <class F>
struct ParamView {
  const GenzParams& p;
  __device__ __forceinline__ auto axis(int i) const { return F::axis_of(p, i); }
};

template <class F>
struct ParamSource {
  const GenzParams* params;
  __device__ __forceinline__ F get(int k) const { return F::load(params[k]); }
};

// Integrals of different families in one batch (family per integral).
template <int N>
struct MixedSource {
  const GenzParams* params;
  const int* families;
  __device__ __forceinline__ MixedGenz<N> get(int k) const {
    return MixedGenz<N>::make(params[k], families[k]);
  }
};

// Write one region's results (reference classification:
// fail when err / max(epsrel|avg|, epsabs) > 1, GPUQuadPhases.cu:63-74).
__device__ __forceinline__ void store_result(const EngineArgs& a, long long slot,
                                             const RegionResult& r, double epsrel, double epsabs) {
  const double ratio = r.err / max_err(r.avg, epsrel, epsabs);
  a.avg[slot] = r.avg;
  a.err[slot] = r.err;
  a.axis[slot] = r.axis;
  a.active[slot] = ratio > 1;
}

__device__ __forceinline__ void store_padding(const EngineArgs& a, long long slot) {
  a.avg[slot] = 0;
  a.err[slot] = 0;
  a.axis[slot] = 0;
  a.active[slot] = 0;
}

// Evaluate slot `slot` with the K lanes of a group (K <= 32, structured
// point enumeration); lane 0 of the group stores the result.
template <int N, int K, class Src>
__device__ __forceinline__ void eval_slot(const Src& src, const RuleTables& T,
                                          const EngineArgs& a, long long slot, int lane,
                                          unsigned gmask, const ItemTable<N>& tab) {
  const int k = a.rid[slot];
  if (k < 0) {
    if (lane == 0) store_padding(a, slot);
    return;
  }
  double L[N], H[N];
#pragma unroll
  for (int d = 0; d < N; ++d) {
    L[d] = a.lo[(long long)d * a.cap + slot];
    H[d] = a.len[(long long)d * a.cap + slot];
  }
  const auto f = src.get(k);
  RegionSums rs;
  region_point_sums<N, K>(f, L, H, lane, tab, T.ratio, rs);
  if (K > 1) reduce_lanes<K>(rs, gmask);
  if (lane == 0) {
    double jac = 1;
#pragma unroll
    for (int d = 0; d < N; ++d) jac = __dmul_rn(jac, H[d]);
    store_result(a, slot, finish_region<N>(rs, T, jac, 0), a.ist[k].epsrel, a.ist[k].epsabs);
  }
}

// The integrand type of a source.
template <class Src>
using SourceFn = std::decay_t<decltype(std::declval<const Src&>().get(0))>;

// What the thread-per-region evaluator reads integral k's integrand from:
// a view of its parameter block for axis products of a batch, else the
// functor.
template <class Src>
__device__ __forceinline__ decltype(auto) source_view(const Src& src, int k) {
  return src.get(k);
}
template <class F>
__device__ __forceinline__ auto source_view(const ParamSource<F>& src, int k) {
  if constexpr (AxisProductTrait<F>::value)
    return ParamView<F>{src.params[k]};
  else
    return src.get(k);
}

// Chunk c's partial from its 32 lanes' values (a padding slot holds zeros
// and is not active); lane 0 stores it.
__device__ __forceinline__ void store_chunk(const EngineArgs& a, long long c, int lane, double av,
                                            double er, bool act) {
  double s0 = av, s1 = er, s2 = act ? 0.0 : av, s3 = act ? 0.0 : er;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, off);
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    s3 += __shfl_xor_sync(0xffffffffu, s3, off);
  }
  const unsigned b = __ballot_sync(0xffffffffu, act);
  if (lane == 0) {
    ChunkPartial p;
    p.sum_avg = s0;
    p.sum_err = s1;
    p.fin_avg = s2;
    p.fin_err = s3;
    p.nactive = __popc(b);
    p.mask = b;
    a.part[c] = p;
    if (a.cmask) a.cmask[c] = b;
  }
}

// One thread per region: a warp evaluates the 32 slots of chunk c and sums
// them on the spot, so values and errors never go through memory (24 B a
// region written and read back by a pass of its own before); only the split
// axes are stored, beside the chunk's partial.
template <int N, class Src>
__device__ __forceinline__ void eval_chunk_warp(const Src& src, const RuleTables& T,
                                                const EngineArgs& a, long long c, int lane,
                                                const ItemTable<N>& tab) {
  const long long slot = c * 32 + lane;
  const int k = a.rid[slot];
  double av = 0, er = 0;
  bool act = false;
  if (k >= 0) {
    RegionSums rs;
    double jac;
    const ListBox box{a.lo + slot, a.len + slot, a.cap};
    const auto& f = source_view(src, k);
    thread_sums<N, SourceFn<Src>>(f, box, tab, T.ratio, rs, jac);
    const RegionResult r = finish_region<N>(rs, T, jac, 0);
    av = r.avg;
    er = r.err;
    act = er / max_err(av, a.ist[k].epsrel, a.ist[k].epsabs) > 1;
    a.axis[slot] = r.axis;
  }
  __syncwarp();
  store_chunk(a, c, lane, av, er, act);
}

// A warp sums the 32 slots of chunk c into a.part[c].
__device__ __forceinline__ void chunk_partial_warp(const EngineArgs& a, long long c, int lane) {
  const long long i = c * 32 + lane;
  const bool valid = i < a.n && a.rid[i] >= 0;
  const double av = valid ? a.avg[i] : 0.0, er = valid ? a.err[i] : 0.0;
  const bool act = valid && a.active[i];
  store_chunk(a, c, lane, av, er, act);
}

// A warp sums the whole tile (if any) that starts within the absolute
// chunks [kTileChunks w, kTileChunks (w + 1)): a.tile[w], and the active
// counts before each of its chunks, from the tile's start, to chunk_excl.
// Such a tile's integral owns the last chunk of that range, so there is one
// at most.  Tiles are counted from the segment's start, so an integral's
// sums do not depend on where its segment lies.
__device__ __forceinline__ void tile_sum_warp(const EngineArgs& a, long long w, int lane) {
  constexpr int kPer = kTileChunks / 32;
  const int k = a.rid[(kTileChunks * w + kTileChunks - 1) * 32];
  const int c0 = a.ist[k].seg_start / 32, nc = (a.ist[k].seg_count + 31) / 32;
  const long long t = w - c0 / kTileChunks;
  if (t < 0 || kTileChunks * (t + 1) > nc) return;
  const long long s = c0 + kTileChunks * t;
  double v0[kPer], v1[kPer], v2[kPer], v3[kPer];
  int na[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const ChunkPartial& p = a.part[s + 32 * i + lane];
    v0[i] = p.sum_avg;
    v1[i] = p.sum_err;
    v2[i] = p.fin_avg;
    v3[i] = p.fin_err;
    na[i] = p.nactive;
  }
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  int run = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    s0 += v0[i];
    s1 += v1[i];
    s2 += v2[i];
    s3 += v3[i];
    int incl = na[i];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += u;
    }
    a.chunk_excl[s + 32 * i + lane] = run + incl - na[i];
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, off);
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    s3 += __shfl_xor_sync(0xffffffffu, s3, off);
  }
  if (lane == 0) {
    TileSum o;
    o.sum_avg = s0;
    o.sum_err = s1;
    o.fin_avg = s2;
    o.fin_err = s3;
    o.nactive = run;
    o.base = 0;
    a.tile[w] = o;
  }
}

// Stop decision for one running integral from the sums of its chunks and
// its active-region count m (GPUKernelquad.cu:565-605).  Sets the child
// count (next_count) or the leftover count (left_new) of phase 2.
__device__ __forceinline__ void decide_integral(IntegralState& is, double s0, double s1, double s2,
                                                double s3, int m, const EngineArgs& a) {
  const double rG = is.value + s0, errG = is.error + s1;
  is.value += s2;
  is.error += s3;
  is.last_value = rG;
  is.last_error = errG;
  is.nregions += (unsigned long long)is.seg_count;
  is.neval += (unsigned long long)is.seg_count * (unsigned long long)a.npoints;
  is.iters += 1;
  is.next_count = 0;
  is.left_new = 0;
  if (!isfinite(s0) || !isfinite(s1)) {
    // a NaN or infinite integrand value reached the sums: stop here
    is.value = rG;
    is.error = errG;
    is.state = kStateDone;
    is.status = kStatusNonFinite;
  } else if (errG <= max_err(rG, is.epsrel, is.epsabs)) {
    // global stop test (GPUKernelquad.cu:583-598)
    is.value = rG;
    is.error = errG;
    is.state = kStateDone;
    is.status = 0;
  } else if (m == 0) {
    // every region finished on its own tolerance
    is.state = kStateDone;
    is.status = 0;
  } else {
    const long long children = 2ll * m;
    const bool cap_hit = a.phase1_cap > 0 && children >= a.phase1_cap;
    const bool iter_hit = is.iters >= a.max_iters;
    if (cap_hit || iter_hit) {
      if (a.policy == kPolicyReference) {
        is.state = kStatePhase2;
        is.left_new = (int)children;
      } else {
        is.state = kStateCapacity;
        is.value = rG;
        is.error = errG;
        is.status = 1;
      }
    } else {
      is.next_count = (int)children;
    }
  }
}

// A warp combines integral k's chunk partials, writes the exclusive scan
// of active counts over its chunks, and takes the stop decision
// (GPUKernelquad.cu:565-605).  With tiles (a.tile), whole tiles of the
// integral come summed already (tile_sum_warp) and only the chunks after
// the last one are read: one warp walking every chunk took 4 ms for the
// 130 k chunks of a 4 M region integral, a fifth of the time of a batch
// that has one such integral.
__device__ __forceinline__ void decide_warp(const EngineArgs& a, int k, int lane) {
  IntegralState& is = a.ist[k];
  if (is.state != kStateRunning) {
    if (lane == 0) {
      is.next_count = 0;
      is.left_new = 0;
    }
    return;
  }
  const int c0 = is.seg_start / 32;
  const int nc = (is.seg_count + 31) / 32;
  const int nt = a.tile ? nc / kTileChunks : 0;
  TileSum* tile = a.tile + (nt ? c0 / kTileChunks : 0);
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
  for (int t = lane; t < nt; t += 32) {
    const TileSum p = tile[t];
    s0 += p.sum_avg;
    s1 += p.sum_err;
    s2 += p.fin_avg;
    s3 += p.fin_err;
  }
  for (int c = nt * kTileChunks + lane; c < nc; c += 32) {
    const ChunkPartial p = a.part[c0 + c];
    s0 += p.sum_avg;
    s1 += p.sum_err;
    s2 += p.fin_avg;
    s3 += p.fin_err;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, off);
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    s3 += __shfl_xor_sync(0xffffffffu, s3, off);
  }
  int running = 0;
  for (int base = 0; base < nt; base += 32) {
    const int t = base + lane;
    const int v = t < nt ? tile[t].nactive : 0;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += u;
    }
    if (t < nt) tile[t].base = running + incl - v;
    running += __shfl_sync(0xffffffffu, incl, 31);
  }
  for (int base = nt * kTileChunks; base < nc; base += 32) {
    const int c = base + lane;
    const int v = c < nc ? a.part[c0 + c].nactive : 0;
    int incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    if (c < nc) a.chunk_excl[c0 + c] = running + incl - v;
    running += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) decide_integral(is, s0, s1, s2, s3, running, a);
}

// One block of kScanThreads assigns the next segments (32-aligned) and the
// leftover ranges of all integrals: an exclusive scan in integral order, an
// integral per thread (a single warp took 10 us for 300 integrals).
constexpr int kScanThreads = 512;
__device__ __forceinline__ void scan_block(const EngineArgs& a, int n_left_in, IterState* out) {
  __shared__ int wn[kScanThreads / 32], wl[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry_n = 0, carry_l = n_left_in, nrun = 0;
  for (int base = 0; base < a.nint; base += kScanThreads) {
    const int k = base + threadIdx.x;
    int vn = 0, vl = 0, r = 0;
    if (k < a.nint) {
      const IntegralState& is = a.ist[k];
      vn = is.state == kStateRunning ? (is.next_count + 31) & ~31 : 0;
      vl = is.left_count == 0 ? is.left_new : 0;  // each integral hands off once
      r = is.state == kStateRunning && is.next_count > 0;
    }
    int in = vn, il = vl;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int tn = __shfl_up_sync(0xffffffffu, in, off);
      const int tl = __shfl_up_sync(0xffffffffu, il, off);
      if (lane >= off) {
        in += tn;
        il += tl;
      }
    }
    if (lane == 31) {
      wn[warp] = in;
      wl[warp] = il;
    }
    nrun += __syncthreads_count(r);
    int pn = carry_n, pl = carry_l;
    for (int w = 0; w < kScanThreads / 32; ++w) {
      if (w < warp) {
        pn += wn[w];
        pl += wl[w];
      }
      carry_n += wn[w];
      carry_l += wl[w];
    }
    if (k < a.nint) {
      IntegralState& is = a.ist[k];
      is.next_start = pn + in - vn;
      if (vl > 0) {
        is.left_start = pl + il - vl;
        is.left_count = vl;
      }
    }
    __syncthreads();  // wn and wl are read before the next pass writes them
  }
  if (threadIdx.x == 0) {
    IterState s;
    s.n = carry_n;
    s.n_running = nrun;
    s.n_left = carry_l;
    s.overflow = (carry_n > a.ncap) || (carry_l > a.left_cap);
    s.handoff = 0;
    *out = s;
  }
}

// A warp writes the children of chunk c's active regions: two adjacent
// children per region, halved on its split axis, to the next list (running
// integrals) or the leftover list (integrals just handed to phase 2).
template <int N>
__device__ __forceinline__ void split_chunk_warp(const EngineArgs& a, long long c, int lane) {
  const ChunkPartial* part = a.part + c;
  const unsigned b = part->mask;
  if (!b) return;
  // a chunk belongs to one integral, and its first slot is never padding
  const int k = a.rid[c * 32];
  const IntegralState& is = a.ist[k];
  const int state = is.state;
  const bool next = state == kStateRunning && is.next_count > 0;
  if (!next && !(state == kStatePhase2 && is.left_new > 0)) return;
  if (!((b >> lane) & 1u)) return;
  const long long i = c * 32 + lane;
  int rank = a.chunk_excl[c] + __popc(b & ((1u << lane) - 1u));
  const int c0 = is.seg_start / 32, nt = (is.seg_count + 31) / 32 / kTileChunks;
  const int t = (int)(c - c0) / kTileChunks;
  if (t < nt) rank += a.tile[c0 / kTileChunks + t].base;
  const int ax = a.axis[i];
  double* dlo;
  double* dlen;
  int* drid;
  long long dcap, dst;
  if (!next) {
    dlo = a.left_lo;
    dlen = a.left_len;
    drid = a.left_rid;
    dcap = a.left_cap;
    dst = is.left_start + 2ll * rank;
  } else {
    dlo = a.nlo;
    dlen = a.nlen;
    drid = a.nrid;
    dcap = a.ncap;
    dst = is.next_start + 2ll * rank;
  }
  // dst and the capacities are even: the children of a region are stored as
  // one 16-byte pair per axis
#pragma unroll
  for (int d = 0; d < N; ++d) {
    const double l = a.lo[(long long)d * a.cap + i];
    const double w = a.len[(long long)d * a.cap + i];
    const double h = d == ax ? w / 2 : w;
    *reinterpret_cast<double2*>(dlo + (long long)d * dcap + dst) =
        make_double2(l, d == ax ? l + 1 * h : l);
    *reinterpret_cast<double2*>(dlen + (long long)d * dcap + dst) = make_double2(h, h);
  }
  *reinterpret_cast<int2*>(drid + dst) = make_int2(k, k);
}

// Padding ids of integral k's next segment, and the segment hand-over
// (the next list becomes current).  A stopped integral's empty segment keeps
// its place among the others: the replicated kernel, which may take the list
// over from here, finds a slot's owner as the last integral that starts at or
// before it (rep_slot_owner).  With the segment left where it was, such an
// integral owned slots of the running ones.
__device__ __forceinline__ void finish_integral(const EngineArgs& a, int k) {
  IntegralState& is = a.ist[k];
  if (is.next_count > 0) {
    const int padded = (is.next_count + 31) & ~31;
    for (int j = is.next_count; j < padded; ++j) a.nrid[is.next_start + j] = -1;
  }
  is.seg_start = is.next_start;
  if (is.state == kStateRunning) {
    is.seg_count = is.next_count;
    if (is.next_count == 0) is.state = kStateDone;
  } else {
    is.seg_count = 0;
  }
}

}  // namespace detail

// ---------------------------------------------------------------------------
// Multi-launch driver kernels (one launch per step).
// ---------------------------------------------------------------------------
// Threads of a block of the rule kernel with K lanes per region, and blocks
// per SM.  Point by point: two blocks of 256 (at most 128 registers); the
// kernel is bound by FP64 latency, so warps in flight matter more than a few
// spilled values.
template <int K, class F>
constexpr int kEvalThreads = K == 1 && detail::kFactored<F> ? 128 : 256;
template <int K, class F>
constexpr int kEvalMinBlocks = K == 1 && detail::kFactored<F> ? 4 : 2;

template <int N, int K, class Src>
__device__ __forceinline__ void eval_list(const Src& src, const RuleTables& T, const EngineArgs& a,
                                          const detail::ItemTable<N>& tab) {
  const int lane = threadIdx.x % (K == 1 ? 32 : K);
  if constexpr (K == 1) {
    const long long nchunk = a.n / 32, nwarp = (long long)gridDim.x * (blockDim.x / 32);
    for (long long c = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; c < nchunk;
         c += nwarp)
      detail::eval_chunk_warp<N>(src, T, a, c, lane, tab);
  } else {
    constexpr int kGroups = 256 / K;
    const unsigned gmask =
        (K == 32) ? 0xffffffffu : (((1u << (K & 31)) - 1u) << ((threadIdx.x & 31) & ~(K - 1)));
    for (long long slot = (long long)blockIdx.x * kGroups + threadIdx.x / K; slot < a.n;
         slot += (long long)gridDim.x * kGroups)
      detail::eval_slot<N, K>(src, T, a, slot, lane, gmask, tab);
  }
}

// The rule over the current list.  K = 1 also leaves the chunk partials;
// K = 8 and 32 need k_partials after them.
template <int N, int K, class Src>
__global__ void __launch_bounds__((kEvalThreads<K, detail::SourceFn<Src>>),
                                  (kEvalMinBlocks<K, detail::SourceFn<Src>>))
    k_eval(Src src, RuleTables T, EngineArgs a) {
  __shared__ detail::ItemTable<N> tab;
  if (!(K == 1 && detail::kFactored<detail::SourceFn<Src>>)) {
    if (threadIdx.x == 0) tab.fill();
    __syncthreads();
  }
  eval_list<N, K>(src, T, a, tab);
}

static __global__ void __launch_bounds__(256) k_partials(EngineArgs a) {
  const long long nchunk = (a.n + 31) / 32;
  for (long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32; c < nchunk;
       c += (long long)gridDim.x * blockDim.x / 32)
    detail::chunk_partial_warp(a, c, threadIdx.x & 31);
}

static __global__ void __launch_bounds__(128) k_tiles(EngineArgs a) {
  const long long nw = a.n / (32 * kTileChunks);
  for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32; w < nw;
       w += (long long)gridDim.x * blockDim.x / 32)
    detail::tile_sum_warp(a, w, threadIdx.x & 31);
}

static __global__ void __launch_bounds__(256) k_decide(EngineArgs a) {
  for (int k = (blockIdx.x * blockDim.x + threadIdx.x) / 32; k < a.nint;
       k += gridDim.x * blockDim.x / 32)
    detail::decide_warp(a, k, threadIdx.x & 31);
}

static __global__ void __launch_bounds__(detail::kScanThreads) k_scan(EngineArgs a) {
  const int n_left = a.ctl->host.n_left;
  __syncthreads();  // the block's last step overwrites it
  detail::scan_block(a, n_left, &a.ctl->host);
}

template <int N>
__global__ void __launch_bounds__(256) k_split(EngineArgs a) {
  if (a.ctl->host.overflow) return;
  const long long nchunk = (a.n + 31) / 32;
  const long long gwarp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const long long nwarp = (long long)gridDim.x * blockDim.x / 32;
  for (long long c = gwarp; c < nchunk; c += nwarp) detail::split_chunk_warp<N>(a, c, threadIdx.x & 31);
}

static __global__ void k_advance(EngineArgs a) {
  if (a.ctl->host.overflow) return;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.nint; k += gridDim.x * blockDim.x)
    detail::finish_integral(a, k);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.ctl->cur ^= 1;
    a.ctl->iters_done += 1;
  }
}

// Slot t of the initial grid: integral t / padded, cell t % padded of the
// d^N equal boxes of its integration box (box[k] = lo[N] then hi[N]; the
// unit cube when box is null), dimension 0 varying fastest
// (GPUKernelquad.cu:24-61,300-316).  Returns the integral, or -1 for a
// padding slot.
template <int N>
__device__ __forceinline__ int initial_box(long long t, int divisions, int per_integral,
                                           int padded, const double* box, double (&L)[N],
                                           double (&H)[N]) {
  const int k = (int)(t / padded);
  const int j = (int)(t % padded);
  if (j >= per_integral) return -1;
  int rem = j;
  const double* bx = box ? box + (long long)k * 2 * N : nullptr;
#pragma unroll
  for (int d = 0; d < N; ++d) {
    const int id = rem % divisions;
    rem /= divisions;
    const double blo = bx ? bx[d] : 0.0;
    const double w = (bx ? bx[N + d] - bx[d] : 1.0) / divisions;
    L[d] = blo + id * w;
    H[d] = w;
  }
  return k;
}

// Initial grid for every integral, written to the current list.
template <int N>
__global__ void k_init_grid(EngineArgs a, int divisions, int per_integral, int padded,
                            const double* box) {
  const long long total = (long long)a.nint * padded;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    double L[N], H[N];
    const int k = initial_box<N>(t, divisions, per_integral, padded, box, L, H);
    if (k >= 0) {
#pragma unroll
      for (int d = 0; d < N; ++d) {
        const_cast<double*>(a.lo)[(long long)d * a.cap + t] = L[d];
        const_cast<double*>(a.len)[(long long)d * a.cap + t] = H[d];
      }
    }
    const_cast<int*>(a.rid)[t] = k;
  }
}

}  // namespace cubature
