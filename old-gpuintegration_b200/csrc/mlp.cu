// mlp.cu -- C ABI of the control-variate network's tensor-core kernels
// (include/cubature/mlp.cuh, umma.cuh).
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>
#include <vector>

#include "capi_internal.h"
#include "cubature/mlp.cuh"

using namespace cubature;
using namespace cubature::capi;

namespace {

int* error_flag() {
  // one device flag per process and device, set by a kernel whose bounded
  // wait gave up
  static int* flags[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  dev &= 63;
  if (!flags[dev]) {
    if (cudaMalloc(&flags[dev], sizeof(int)) != cudaSuccess) return nullptr;
    cudaMemset(flags[dev], 0, sizeof(int));
  }
  return flags[dev];
}

// Allow `kernel` its dynamic shared memory, once per device.
template <class K>
cudaError_t allow_smem(K kernel, int bytes, std::atomic<bool> (&done)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (done[dev & 63].load(std::memory_order_relaxed)) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[dev & 63].store(true, std::memory_order_relaxed);
  return e;
}

template <int N>
cudaError_t launch_gemm(dim3 grid, cudaStream_t s, const umma::GemmArgs& g, float* out,
                        long long ld_out, long long batch_out) {
  static std::atomic<bool> configured[64];
  const cudaError_t e = allow_smem(mlp::k_gemm<N>, mlp::kGemmSmem, configured);
  if (e != cudaSuccess) return e;
  mlp::k_gemm<N><<<grid, 128, mlp::kGemmSmem, s>>>(g, out, ld_out, batch_out);
  return cudaGetLastError();
}

template <bool kTrain>
cudaError_t launch_net(dim3 grid, cudaStream_t s, const mlp::NetArgs& a) {
  static std::atomic<bool> configured[64];
  const cudaError_t e = allow_smem(mlp::k_net<kTrain>, mlp::kNetSmem<kTrain>, configured);
  if (e != cudaSuccess) return e;
  mlp::k_net<kTrain><<<grid, mlp::kNetThreads, mlp::kNetSmem<kTrain>, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

int cub_mlp_gemm_bf16(int batch, int m, int n, int k, const void* d_a, long long lda,
                      const void* d_b, long long ldb, float* d_d, long long ldd, void* stream) {
  if (batch <= 0 || m <= 0 || m % umma::kTileM || k <= 0 || k % 16 || (n != 16 && n != 128) ||
      !d_a || !d_b || !d_d || lda < k || ldb < k || ldd < n || lda % 8 || ldb % 8) {
    set_error("cub_mlp_gemm_bf16: m % 128, k % 16, n in {16, 128}, lda/ldb % 8 required");
    return CUB_ERR_INVALID;
  }
  int* err = error_flag();
  if (!err) return cuda_error(cudaErrorMemoryAllocation, "error flag");
  cudaStream_t s = as_stream(stream);
  umma::GemmArgs g;
  g.a = static_cast<const __nv_bfloat16*>(d_a);
  g.b = static_cast<const __nv_bfloat16*>(d_b);
  g.lda = lda;
  g.ldb = ldb;
  g.batch_a = lda * m;
  g.batch_b = ldb * n;
  g.m = m;
  g.k = k;
  g.error = err;
  const dim3 grid(m / umma::kTileM, 1, batch);
  cudaError_t e;
  if (n == 16) {
    e = launch_gemm<16>(grid, s, g, d_d, ldd, ldd * m);
  } else {
    e = launch_gemm<128>(grid, s, g, d_d, ldd, ldd * m);
  }
  if (e != cudaSuccess) return cuda_error(e, "k_gemm launch");
  int h_err = 0;
  if ((e = cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return cuda_error(e, "k_gemm");
  if (h_err) {
    cudaMemsetAsync(err, 0, sizeof(int), s);
    set_error("tensor-core GEMM: a bounded wait gave up");
    return CUB_ERR_TIMEOUT;
  }
  return 0;
}

// ---------------------------------------------------------------------------
// The networks: buffers, training and inference.
// ---------------------------------------------------------------------------
using mlp::Layout;
using bf16 = __nv_bfloat16;

struct cub_mlp {
  int device = 0, E = 0, S = 0, B = 0;
  cudaStream_t stream = nullptr;
  int* err = nullptr;
  int step = 0;
  bool have_data = false;
  void* mem = nullptr;  // the one allocation all buffers are cut from
  float *P, *G, *Mm, *Vv, *part, *loss, *scale, *Y;
  bf16 *W0, *W1, *W1T, *W2, *W2T, *X, *XT;
  bf16 *Z1, *Z2, *H1T, *H2T, *dZ1T, *dZ2T, *dZ3T;

  ~cub_mlp() {
    cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    if (mem) cudaFree(mem);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

int check(cudaError_t e, const char* what) { return e == cudaSuccess ? 0 : cuda_error(e, what); }

mlp::BfWeights bf_weights(const cub_mlp* m) { return {m->W0, m->W1, m->W1T, m->W2, m->W2T}; }

int refresh(cub_mlp* m) {
  mlp::k_refresh_weights<<<592, 256, 0, m->stream>>>(m->P, (long long)m->E * Layout::kCount,
                                                     bf_weights(m));
  return check(cudaGetLastError(), "k_refresh_weights");
}

mlp::NetArgs net_args(const cub_mlp* m) {
  mlp::NetArgs a{};
  a.P = m->P;
  a.W0 = m->W0;
  a.W1 = m->W1;
  a.W2 = m->W2;
  a.W1T = m->W1T;
  a.W2T = m->W2T;
  a.error = m->err;
  return a;
}

// Forward + backward of minibatch b into G (no update); loss into m->loss.
int grad_step(cub_mlp* m, int b) {
  const long long B = m->B, S = m->S, s0 = (long long)b * B;
  const int ntiles = m->B / 128;
  mlp::NetArgs a = net_args(m);
  a.X = m->X + s0 * mlp::kInPad;
  a.batch_X = S * mlp::kInPad;
  a.y = m->Y + s0;
  a.batch_y = S;
  a.inv_nbatch = 1.0f / (float)m->B;
  a.Z1 = m->Z1;
  a.Z2 = m->Z2;
  a.H1T = m->H1T;
  a.H2T = m->H2T;
  a.dZ1T = m->dZ1T;
  a.dZ2T = m->dZ2T;
  a.dZ3T = m->dZ3T;
  a.part = m->part;
  a.rows = B;
  int rc = check(launch_net<true>(dim3(ntiles, 1, m->E), m->stream, a), "k_net");
  if (rc) return rc;
  mlp::GradArgs g{};
  g.dZT[0] = m->dZ1T;
  g.dZT[1] = m->dZ2T;
  g.dZT[2] = m->dZ3T;
  g.HT[0] = m->XT + s0;
  g.HT[1] = m->H1T;
  g.HT[2] = m->H2T;
  g.ldx = S;
  g.rows = B;
  g.G = m->G;
  g.error = m->err;
  static std::atomic<bool> configured[64];
  rc = check(allow_smem(mlp::k_weight_grads, mlp::kGradSmem, configured), "k_weight_grads");
  if (rc) return rc;
  mlp::k_weight_grads<<<dim3(3, 1, m->E), 128, mlp::kGradSmem, m->stream>>>(g);
  if ((rc = check(cudaGetLastError(), "k_weight_grads"))) return rc;
  mlp::k_small_grads<<<dim3(49, 1, m->E), 256, 0, m->stream>>>(g, m->part, ntiles, m->loss,
                                                               a.inv_nbatch);
  return check(cudaGetLastError(), "k_small_grads");
}

int read_error(cub_mlp* m) {
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return cuda_error(e, "network kernels");
  if (h) {
    cudaMemsetAsync(m->err, 0, sizeof(int), m->stream);
    set_error("tensor-core GEMM: a bounded wait gave up");
    return CUB_ERR_TIMEOUT;
  }
  return 0;
}

}  // namespace

cub_mlp* cub_mlp_create(int device, int count, int samples, int batch, unsigned long long seed) {
  if (count <= 0 || batch <= 0 || batch % 128 || samples <= 0 || samples % batch) {
    set_error("cub_mlp_create: batch a multiple of 128 and samples a multiple of batch");
    return nullptr;
  }
  if (cudaSetDevice(device) != cudaSuccess) {
    set_error("cudaSetDevice failed");
    return nullptr;
  }
  auto* m = new cub_mlp;
  m->device = device;
  m->E = count;
  m->S = samples;
  m->B = batch;
  const size_t E = count, S = samples, B = batch, P = Layout::kCount;
  // one allocation, cut into 256-byte aligned buffers (a create and destroy
  // of 38 allocations cost milliseconds); a first pass adds the sizes up
  char* base = nullptr;
  size_t used = 0;
  auto cut = [&](auto** p, size_t n) {
    *p = reinterpret_cast<std::remove_pointer_t<decltype(p)>>(base + used);
    used += (n * sizeof(**p) + 255) & ~size_t(255);
  };
  auto layout = [&] {
    used = 0;
    cut(&m->err, 1);
    for (float** q : {&m->P, &m->G, &m->Mm, &m->Vv}) cut(q, E * P);
    cut(&m->part, E * (B / 128) * (128 + 2));
    cut(&m->loss, E);
    cut(&m->scale, E);
    cut(&m->Y, E * S);
    cut(&m->W0, E * 128 * 16);
    for (bf16** q : {&m->W1, &m->W1T, &m->W2, &m->W2T}) cut(q, E * 128 * 128);
    cut(&m->X, E * S * 16);
    cut(&m->XT, E * S * 16);
    for (bf16** q : {&m->Z1, &m->Z2, &m->H1T, &m->H2T, &m->dZ1T, &m->dZ2T, &m->dZ3T})
      cut(q, E * B * 128);
  };
  layout();
  bool ok = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMalloc(&m->mem, used) == cudaSuccess;
  base = static_cast<char*>(m->mem);
  if (ok) layout();
  if (!ok) {
    set_error("cub_mlp_create: device allocation failed");
    delete m;
    return nullptr;
  }
  const long long runs = ((long long)count * mlp::kInitDraws + mlp::kInitRun - 1) / mlp::kInitRun;
  ok = cudaMemsetAsync(m->err, 0, sizeof(int), m->stream) == cudaSuccess;
  for (float* q : {m->P, m->G, m->Mm, m->Vv})
    ok = ok && cudaMemsetAsync(q, 0, sizeof(float) * E * P, m->stream) == cudaSuccess;
  if (ok) {
    mlp::k_init_params<<<(unsigned)((runs + 127) / 128), 128, 0, m->stream>>>(
        m->P, count, seed * mlp::kLcgA + mlp::kLcgC);
    ok = cudaGetLastError() == cudaSuccess && refresh(m) == 0 &&
         cudaStreamSynchronize(m->stream) == cudaSuccess;
  }
  if (!ok) {
    set_error("cub_mlp_create: initialisation failed");
    delete m;
    return nullptr;
  }
  return m;
}

void cub_mlp_destroy(cub_mlp* m) { delete m; }

int cub_mlp_set_data(cub_mlp* m, const double* d_x, const double* d_y) {
  if (!m || !d_x || !d_y) {
    set_error("invalid argument");
    return CUB_ERR_INVALID;
  }
  cudaSetDevice(m->device);
  const long long S = m->S;
  mlp::k_prep_inputs<<<dim3(64, 1, m->E), 256, 0, m->stream>>>(d_x, S, S * mlp::kIn, m->X, m->XT,
                                                                 S, S * mlp::kInPad,
                                                                 S * mlp::kInPad);
  mlp::k_scale_targets<<<dim3(1, 1, m->E), 256, 0, m->stream>>>(d_y, S, m->Y, m->scale);
  int rc = check(cudaGetLastError(), "set_data");
  if (!rc) rc = check(cudaStreamSynchronize(m->stream), "set_data");
  m->have_data = rc == 0;
  return rc;
}

int cub_mlp_params(cub_mlp* m, float* h_params, int set) {
  if (!m || !h_params) {
    set_error("invalid argument");
    return CUB_ERR_INVALID;
  }
  cudaSetDevice(m->device);
  const size_t bytes = sizeof(float) * (size_t)m->E * Layout::kCount;
  int rc = set ? check(cudaMemcpyAsync(m->P, h_params, bytes, cudaMemcpyHostToDevice, m->stream),
                       "params")
               : check(cudaMemcpyAsync(h_params, m->P, bytes, cudaMemcpyDeviceToHost, m->stream),
                       "params");
  if (!rc && set) rc = refresh(m);
  if (!rc) rc = check(cudaStreamSynchronize(m->stream), "params");
  return rc;
}

int cub_mlp_grad(cub_mlp* m, int b, float* h_loss, float* h_grads) {
  if (!m || !m->have_data || b < 0 || b >= m->S / m->B) {
    set_error("cub_mlp_grad: no data or minibatch out of range");
    return CUB_ERR_INVALID;
  }
  cudaSetDevice(m->device);
  int rc = grad_step(m, b);
  if (!rc) rc = read_error(m);
  if (!rc && h_loss)
    rc = check(cudaMemcpy(h_loss, m->loss, sizeof(float) * m->E, cudaMemcpyDeviceToHost), "loss");
  if (!rc && h_grads)
    rc = check(cudaMemcpy(h_grads, m->G, sizeof(float) * (size_t)m->E * Layout::kCount,
                          cudaMemcpyDeviceToHost),
               "grads");
  return rc;
}

int cub_mlp_train(cub_mlp* m, int epochs, float lr, float* h_loss) {
  if (!m || !m->have_data || epochs < 0 || !(lr > 0)) {
    set_error("cub_mlp_train: no data or bad arguments");
    return CUB_ERR_INVALID;
  }
  cudaSetDevice(m->device);
  const int nb = m->S / m->B;
  const long long n = (long long)m->E * Layout::kCount;
  const float b1 = 0.9f, b2 = 0.999f;
  for (int ep = 0; ep < epochs; ++ep) {
    for (int b = 0; b < nb; ++b) {
      int rc = grad_step(m, b);
      if (rc) return rc;
      ++m->step;
      const float c1 = 1.0f - std::pow(b1, (float)m->step), c2 = 1.0f - std::pow(b2, (float)m->step);
      mlp::k_adam<<<592, 256, 0, m->stream>>>(m->P, m->G, m->Mm, m->Vv, n, lr, b1, b2, 1e-8f, c1,
                                              c2, bf_weights(m));
      if ((rc = check(cudaGetLastError(), "k_adam"))) return rc;
    }
    int rc = read_error(m);  // once per epoch
    if (rc) return rc;
  }
  if (h_loss)
    return check(cudaMemcpy(h_loss, m->loss, sizeof(float) * m->E, cudaMemcpyDeviceToHost), "loss");
  return 0;
}

int cub_mlp_eval(cub_mlp* m, long long n, const double* d_x, double* d_g) {
  if (!m || n <= 0 || !d_x || !d_g) {
    set_error("invalid argument");
    return CUB_ERR_INVALID;
  }
  cudaSetDevice(m->device);
  mlp::NetArgs a = net_args(m);
  a.x = d_x;
  a.n = n;
  a.scale = m->scale;
  a.g = d_g;
  // two blocks fit on an SM; a block keeps its network's weights and walks
  // over tiles
  const long long tiles = (n + 127) / 128;
  const long long blocks =
      std::min<long long>(tiles, std::max(1, (2 * sm_count(m->device) + m->E - 1) / m->E));
  const int rc = check(launch_net<false>(dim3((unsigned)blocks, 1, m->E), m->stream, a), "k_net");
  if (rc) return rc;
  return read_error(m);
}

// ---------------------------------------------------------------------------
// Learned control variate: integral of f = integral of g + integral of
// (f - g), with g the network trained on f's values at rule nodes.
// ---------------------------------------------------------------------------
#include "cubature/engine.cuh"

namespace {

constexpr int kCvDim = 7;
using CvPT = detail::PointTable<kCvDim>;

// f at points x [E][S][7] for integral e's parameters -> y [E][S].
template <class F>
__global__ void k_eval_points(const GenzParams* params, const double* x, long long S, double* y) {
  const int e = blockIdx.z;
  const F f = F::load(params[e]);
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < S;
       s += (long long)gridDim.x * blockDim.x)
    y[e * S + s] = f(x + (e * S + s) * kCvDim);
}

// a f(x) + b g_p at the rule points of one region (g_p precomputed).
template <class F>
struct CvPoint {
  F f;
  double a, b;
  const double* g;
  __device__ __forceinline__ double operator()(const double* x, int p) const {
    const double gv = g[p];
    return a != 0.0 ? a * f(x) + b * gv : b * gv;
  }
};

// Rule and fourth difference of slots [0, n) for the integrand a f + b g:
// eight regions per block, 32 threads each.  A region stays active while
// its error exceeds its volume's share of the absolute budget,
// err > budget * volume (unit-cube volume 1), so that when every region is
// finished the total error is within the budget.
template <class F>
__global__ void __launch_bounds__(256) k_eval_cv(F f, double ca, double cb, const double* g,
                                                 RuleTables T, EngineArgs a, long long s0,
                                                 long long n, double budget) {
  __shared__ detail::GroupSmem<kCvDim> sm;
  sm.pt.fill(threadIdx.x, blockDim.x);
  __syncthreads();
  const int grp = threadIdx.x / 32, t = threadIdx.x % 32;
  const long long ngroups = 8ll * gridDim.x;
  for (long long base = 0; base < n; base += ngroups) {
    const long long local = base + (long long)grp * gridDim.x + blockIdx.x;
    const bool live = local < n;
    const long long slot = s0 + local;
    const int k = live ? a.rid[slot] : -1;
    double L[kCvDim], H[kCvDim];
#pragma unroll
    for (int d = 0; d < kCvDim; ++d) {
      L[d] = k >= 0 ? a.lo[(long long)d * a.cap + slot] : 0.0;
      H[d] = k >= 0 ? a.len[(long long)d * a.cap + slot] : 1.0;
    }
    const CvPoint<F> h{f, ca, cb, g + (k >= 0 ? local : 0) * CvPT::kPoints};
    const detail::RegionResult r =
        detail::eval_region_group<kCvDim, 32>(h, L, H, T, sm, grp, t, k >= 0);
    if (t == 0 && live) {
      if (k >= 0) {
        double vol = 1;
#pragma unroll
        for (int d = 0; d < kCvDim; ++d) vol *= H[d];
        a.avg[slot] = r.avg;
        a.err[slot] = r.err;
        a.axis[slot] = r.axis;
        a.active[slot] = r.err > budget * vol;
      } else {
        detail::store_padding(a, slot);
      }
    }
  }
}

// The network as a smooth function for integration: its bf16 weights with
// FP32 activations and FP32 arithmetic on the CUDA cores (the tensor-core
// path rounds every activation to bf16, a quantisation of ~2^-8 relative
// that no bisection resolves, so an adaptive rule cannot converge on it).
// 128 nodes per block at a time: the weights sit transposed in shared memory
// (W^T[in][out]), the nodes' activations beside them ([unit][node]), and a
// thread accumulates 8 nodes x 8 units in registers, so a unit step costs it
// four 16-byte loads for 64 FMAs (a warp per node reloaded every weight for
// every node: 24.4 M nodes took 130 ms, bound by shared memory).  Each sum
// runs over the inputs in order, starting from the bias.  g[r] for the nodes
// of slots [s0, s0 + n), row (s - s0) * npts + p.
constexpr int kSmoothNodes = 128;
constexpr int kSmoothLd = kSmoothNodes + 4;  // row of the activations (16-byte aligned)
constexpr int kSmoothSmem =
    (16 * 128 + 2 * 128 * 128 + 4 * 128 + 128 * kSmoothLd + 8 * kSmoothNodes) * 4;

// Two FP32 FMAs in one instruction (each rounded as fmaf).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)),
        "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}

// acc[node][unit pair] += W^T[i][unit] * h[i][node], i = 0 .. n-1 in order, for
// nodes 0..3 and 64..67 of h and units 0..3 and 64..67 of wt (16-byte loads of
// neighbouring threads are then contiguous).
__device__ __forceinline__ void smooth_layer(float2 (&acc)[8][4], const float* wt, const float* h,
                                             int ld, int n) {
#pragma unroll 4
  for (int i = 0; i < n; ++i) {
    const float4 a0 = *reinterpret_cast<const float4*>(h + i * ld);
    const float4 a1 = *reinterpret_cast<const float4*>(h + i * ld + 64);
    const float4 b0 = *reinterpret_cast<const float4*>(wt + i * 128);
    const float4 b1 = *reinterpret_cast<const float4*>(wt + i * 128 + 64);
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float2 b[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w),
                         make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = fma2(b[q], make_float2(a[p], a[p]), acc[p][q]);
  }
}

__global__ void __launch_bounds__(256) k_cv_smooth(const float* P, const bf16* W0, const bf16* W1,
                                                   const bf16* W2, float scale, const double* lo,
                                                   const double* len, const int* rid,
                                                   long long cap, long long s0, long long n,
                                                   double* g) {
  extern __shared__ __align__(16) float fsm[];
  float* w0t = fsm;                         // [16][128]
  float* w1t = w0t + 16 * 128;              // [128][128]
  float* w2t = w1t + 128 * 128;             // [128][128]
  float* bias = w2t + 128 * 128;            // b0, b1, b2, w3
  float* act = bias + 4 * 128;              // [128 units][kSmoothLd]
  float* xs = act + 128 * kSmoothLd;        // [8 inputs][128 nodes]
  __shared__ CvPT pt;
  pt.fill(threadIdx.x, blockDim.x);
  for (int i = threadIdx.x; i < 128 * 128; i += blockDim.x) {
    const int o = i % 128, in = i / 128;
    w1t[i] = __bfloat162float(W1[o * 128 + in]);
    w2t[i] = __bfloat162float(W2[o * 128 + in]);
    if (i < 128 * 16) w0t[i] = __bfloat162float(W0[o * 16 + in]);
  }
  for (int j = threadIdx.x; j < 128; j += blockDim.x) {
    bias[j] = P[Layout::B0 + j];
    bias[128 + j] = P[Layout::B1 + j];
    bias[256 + j] = P[Layout::B2 + j];
    bias[384 + j] = P[Layout::W3 + j];
  }
  __syncthreads();
  const float b3 = P[Layout::B3];
  const int u0 = (threadIdx.x & 15) * 4, n0 = (threadIdx.x >> 4) * 4;  // this thread's tile
  const long long nodes = n * CvPT::kPoints;
  for (long long base = (long long)blockIdx.x * kSmoothNodes; base < nodes;
       base += (long long)gridDim.x * kSmoothNodes) {
    if (threadIdx.x < kSmoothNodes) {
      const long long r = base + threadIdx.x;
      const long long s = s0 + r / CvPT::kPoints;
      const bool live = r < nodes && rid[s] >= 0;
      const uint2 e = pt.ent[(int)(r % CvPT::kPoints)];
#pragma unroll
      for (int i = 0; i < kCvDim; ++i) {
        const double x = live ? fma(pt.ctab[(e.x >> (4 * i)) & 15u], len[(long long)i * cap + s],
                                    lo[(long long)i * cap + s])
                              : 0.0;
        xs[i * kSmoothNodes + threadIdx.x] = (float)(2.0 * x - 1.0);
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
      float2 acc[8][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float* b = bias + l * 128 + u0 + (q >> 1) * 64 + (q & 1) * 2;
        const float2 b2 = make_float2(b[0], b[1]);
#pragma unroll
        for (int p = 0; p < 8; ++p) acc[p][q] = b2;
      }
      if (l == 0)
        smooth_layer(acc, w0t + u0, xs + n0, kSmoothNodes, kCvDim);
      else
        smooth_layer(acc, (l == 1 ? w1t : w2t) + u0, act + n0, kSmoothLd, 128);
      __syncthreads();  // every thread has read the layer's inputs
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float* d = act + (u0 + (q >> 1) * 64 + (q & 1) * 2) * kSmoothLd + n0;
#pragma unroll
        for (int p = 0; p < 8; ++p)
          acc[p][q] = make_float2(mlp::silu(acc[p][q].x), mlp::silu(acc[p][q].y));
#pragma unroll
        for (int p = 0; p < 8; p += 4) {
          *reinterpret_cast<float4*>(d + p * 16) =
              make_float4(acc[p][q].x, acc[p + 1][q].x, acc[p + 2][q].x, acc[p + 3][q].x);
          *reinterpret_cast<float4*>(d + kSmoothLd + p * 16) =
              make_float4(acc[p][q].y, acc[p + 1][q].y, acc[p + 2][q].y, acc[p + 3][q].y);
        }
      }
      __syncthreads();
    }
    // Output layer, two threads per node: 32 interleaved partial sums of four
    // units each, added as a tree over the partials' index bits from the top
    // (16, 8, 4, 2) down; a thread holds those of one parity.
    {
      const int node = threadIdx.x >> 1, par = threadIdx.x & 1;
      const float* h = act + node;
      const float* w3 = bias + 384;
      float t[16];
#pragma unroll
      for (int v = 0; v < 16; ++v) {
        const int l = 2 * v + par;
        float a = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) a = fmaf(w3[l + 32 * q], h[(l + 32 * q) * kSmoothLd], a);
        t[v] = a;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < 8; ++v)
          if (v < o) t[v] += t[v + o];
      const float sum = t[0] + __shfl_xor_sync(0xffffffffu, t[0], 1);
      const long long r = base + node;
      if (par == 0 && r < nodes)
        g[r] = rid[s0 + r / CvPT::kPoints] < 0 ? 0.0 : (double)scale * (double)(sum + b3);
    }
    __syncthreads();  // the next tile overwrites the activations
  }
}

// Evaluation hook of the engine's multi-launch driver: the rule over the
// current list for a f + b g, g from network net_k at every rule point.
template <class F>
struct CvHook {
  static constexpr bool kActive = true;
  cub_mlp* net;
  int net_k;
  F f;
  double ca, cb;
  double budget;  // absolute error budget of the integral
  RuleTables T;
  int sms;
  // growable scratch (shared by the hook's copies)
  struct Scratch {
    long long rows = 0;
    double* g = nullptr;  // the network at the rule nodes
    void release() {
      cudaFree(g);
      g = nullptr;
      rows = 0;
    }
  };
  Scratch* sc;

  // Node rows per chunk: 32 MB of values, whatever the length of the list.
  static constexpr long long kRowsMax = 1ll << 22;

  int eval(const EngineArgs& a, long long n, cudaStream_t s) const {
    const long long per = kRowsMax / CvPT::kPoints;  // slots per chunk
    const long long cmax = std::min(n, per);
    const long long rmax = (cmax * CvPT::kPoints + 127) / 128 * 128;
    if (rmax > sc->rows) {
      cudaStreamSynchronize(s);
      sc->release();
      const long long r = std::max(rmax, 1ll << 16);
      if (cudaMalloc(&sc->g, sizeof(double) * r) != cudaSuccess) {
        set_error("control variate: scratch allocation failed");
        return kErrCuda;
      }
      sc->rows = r;
    }
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[dev & 63]) {
      if (cudaFuncSetAttribute(k_cv_smooth, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kSmoothSmem) != cudaSuccess)
        return kErrCuda;
      configured[dev & 63] = true;
    }
    float scale = 1.0f;
    cudaMemcpyAsync(&scale, net->scale + net_k, sizeof(float), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    const long long P = Layout::kCount;
    for (long long s0 = 0; s0 < n; s0 += per) {
      const long long cn = std::min(per, n - s0);
      k_cv_smooth<<<(unsigned)sms, 256, kSmoothSmem, s>>>(
          net->P + net_k * P, net->W0 + (long long)net_k * 128 * 16,
          net->W1 + (long long)net_k * 128 * 128, net->W2 + (long long)net_k * 128 * 128, scale,
          a.lo, a.len, a.rid, a.cap, s0, cn, sc->g);
      if (cudaGetLastError() != cudaSuccess) return kErrCuda;
      const long long eb = std::min<long long>((cn + 7) / 8, (long long)sms * 8);
      k_eval_cv<F><<<(unsigned)std::max<long long>(eb, 1), 256, 0, s>>>(f, ca, cb, sc->g, T, a,
                                                                        s0, cn, budget);
      if (cudaGetLastError() != cudaSuccess) return kErrCuda;
    }
    return 0;
  }
};

double now_ms() {
  return std::chrono::duration<double, std::milli>(
             std::chrono::steady_clock::now().time_since_epoch())
      .count();
}

// The whole control-variate flow for one family (N = 7).
template <template <int> class Fam>
int cv_run(cub_ctx* ctx, int count, const GenzParams* h, double epsrel, double epsabs,
           const cub_cv_options& co, cub_result* out, cub_cv_stats* st) {
  using F = Fam<kCvDim>;
  Workspace& ws = *ctx->ws;
  const cudaStream_t s = ctx->stream;
  Options o;
  o.policy = kPolicyBreadth;
  o.max_slots = ws.auto_slots(kCvDim, o.policy);
  const RuleTables T = make_rule9_tables(kCvDim);
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = sm_count(dev);
  std::vector<double> er(count), ea(count);
  std::vector<Result> coarse(count), res(count);
  double t0 = now_ms();

  // 1. coarse plain run: the check of the result and the scale of the tolerances
  GenzParams* d_par = nullptr;
  if (cudaMalloc(&d_par, sizeof(GenzParams) * count) != cudaSuccess)
    return cuda_error(cudaErrorMemoryAllocation, "params");
  std::unique_ptr<GenzParams, decltype(&cudaFree)> par_guard(d_par, cudaFree);
  cudaMemcpyAsync(d_par, h, sizeof(GenzParams) * count, cudaMemcpyHostToDevice, s);
  for (int k = 0; k < count; ++k) {
    er[k] = std::max(co.coarse_epsrel, epsrel);
    ea[k] = epsabs;
  }
  {
    detail::ParamSource<F> src{d_par};
    const int rc = grouped_batch(count, o, [&](const std::vector<int>& idx, Result* g) {
      // groups of the batch run on consecutive parameter blocks
      detail::ParamSource<F> gs{d_par + idx[0]};
      (void)src;
      return run_batch<kCvDim>(ws, gs, (int)idx.size(), er.data(), ea.data(), o, g, s);
    }, coarse);
    if (rc != kOk && rc != kErrCapacity) return engine_status(ctx, rc);
  }
  st->ms_coarse = now_ms() - t0;

  // 2. training data: rule nodes of the initial grid (2^7 boxes), S per
  //    integral drawn with a seeded generator, and f there
  t0 = now_ms();
  const long long S = co.samples;
  std::vector<double> hx((size_t)count * S * kCvDim);
  unsigned long long rs = co.seed * 0x9E3779B97F4A7C15ull + 1;
  auto next = [&rs]() {
    rs = rs * 6364136223846793005ull + 1442695040888963407ull;
    return rs >> 17;
  };
  const double gen[5] = {kGenA1, kGenA2, kGenA3, kGenA4, kGenL};
  for (int e = 0; e < count; ++e)
    for (long long q = 0; q < S; ++q) {
      const int box = (int)(next() % 128), p = (int)(next() % CvPT::kPoints);
      const uint2 en = CvPT::entry(p);
      for (int i = 0; i < kCvDim; ++i) {
        const int c = (en.x >> (4 * i)) & 15;
        const double cf = c == 0 ? 0.5 : detail::coef(gen[(c - 1) >> 1], (c - 1) & 1);
        hx[((size_t)e * S + q) * kCvDim + i] = 0.5 * ((box >> i) & 1) + cf * 0.5;
      }
    }
  double *d_x = nullptr, *d_y = nullptr, *d_g = nullptr;
  if (cudaMalloc(&d_x, sizeof(double) * hx.size()) != cudaSuccess ||
      cudaMalloc(&d_y, sizeof(double) * count * S) != cudaSuccess ||
      cudaMalloc(&d_g, sizeof(double) * count * S) != cudaSuccess)
    return cuda_error(cudaErrorMemoryAllocation, "training data");
  std::unique_ptr<double, decltype(&cudaFree)> gx(d_x, cudaFree), gy(d_y, cudaFree),
      gg(d_g, cudaFree);
  cudaMemcpyAsync(d_x, hx.data(), sizeof(double) * hx.size(), cudaMemcpyHostToDevice, s);
  k_eval_points<F><<<dim3(32, 1, count), 256, 0, s>>>(d_par, d_x, S, d_y);
  if (cudaStreamSynchronize(s) != cudaSuccess) return cuda_error(cudaGetLastError(), "harvest");

  // 3. train the networks
  cub_mlp* net = cub_mlp_create(ctx->device, count, (int)S, co.batch, co.seed);
  if (!net) return CUB_ERR_CUDA;
  std::unique_ptr<cub_mlp, decltype(&cub_mlp_destroy)> net_guard(net, cub_mlp_destroy);
  int rc = cub_mlp_set_data(net, d_x, d_y);
  if (!rc) rc = cub_mlp_train(net, co.epochs, co.lr, nullptr);
  if (!rc) rc = cub_mlp_eval(net, S, d_x, d_g);
  if (rc) return rc;
  std::vector<double> hy((size_t)count * S), hg((size_t)count * S);
  cudaMemcpy(hy.data(), d_y, sizeof(double) * hy.size(), cudaMemcpyDeviceToHost);
  cudaMemcpy(hg.data(), d_g, sizeof(double) * hg.size(), cudaMemcpyDeviceToHost);
  st->ms_train = now_ms() - t0;

  // 4. per integral: residual and network integrals, or the plain method
  t0 = now_ms();
  typename CvHook<F>::Scratch scratch;
  st->fallbacks = 0;
  st->rejected = 0;
  double rho_sum = 0;
  std::vector<int> plain_idx;  // integrals the plain method integrates
  for (int k = 0; k < count; ++k) {
    double num = 0, den = 0;
    for (long long q = 0; q < S; ++q) {
      const double y = hy[(size_t)k * S + q], d = y - hg[(size_t)k * S + q];
      num += d * d;
      den += y * y;
    }
    const double rho = den > 0 ? std::sqrt(num / den) : 1.0;
    rho_sum += rho;
    const double tol = std::max(epsrel * std::fabs(coarse[k].value), epsabs);
    bool use_plain = !(rho <= co.rho_max) || coarse[k].status != 0;
    Result cv{};
    if (!use_plain) {
      const F f = F::load(h[k]);
      detail::SingleSource<F> dummy{f};
      const double half = 0.5 * tol, zero = 0.0;
      Result rr, rg;
      // a residual that does not converge within 2^20 regions (its error
      // estimate has not shrunk to the budget) stops there and the plain
      // method takes over
      Options oc = o;
      oc.max_slots = std::min<long long>(o.max_slots, 1ll << 20);
      CvHook<F> hr{net, k, f, 1.0, -1.0, half, T, sms, &scratch};
      CvHook<F> hgk{net, k, f, 0.0, 1.0, half, T, sms, &scratch};
      int r1 = run_batch<kCvDim>(ws, dummy, 1, &zero, &half, oc, &rr, s, nullptr, hr);
      int r2 = r1 == kOk ? run_batch<kCvDim>(ws, dummy, 1, &zero, &half, oc, &rg, s, nullptr, hgk)
                         : r1;
      if (r1 != kOk && r1 != kErrCapacity) {
        scratch.release();
        return engine_status(ctx, r1);
      }
      if (r2 != kOk && r2 != kErrCapacity) {
        scratch.release();
        return engine_status(ctx, r2);
      }
      if (r1 == kErrCapacity || r2 == kErrCapacity) rr.status = 1;
      st->regions_residual += rr.nregions;
      st->regions_network += rg.nregions;
      cv.value = rr.value + rg.value;
      cv.error = rr.error + rg.error;
      cv.nregions = rr.nregions + rg.nregions;
      cv.neval = rr.neval + rg.neval;
      cv.status = (rr.status || rg.status) ? 1 : 0;
      cv.iterations = rr.iterations + rg.iterations;
      cv.state = kStateDone;
      // the plain coarse run checks the result
      const bool agrees = std::fabs(cv.value - coarse[k].value) <=
                          3.0 * (coarse[k].error + cv.error) + 1e-300;
      if (cv.status != 0 || !agrees) {
        use_plain = true;
        st->rejected += 1;
      }
    }
    if (use_plain) {
      // integrated with the other fallbacks in one batch below
      st->fallbacks += 1;
      plain_idx.push_back(k);
      continue;
    }
    result_to_c(cv, &out[k]);
  }
  scratch.release();
  if (!plain_idx.empty()) {
    // the plain method on every integral that fell back, batched as
    // cub_integrate_batch would run them (groups on consecutive parameter
    // blocks of a staging copy)
    const int np = (int)plain_idx.size();
    GenzParams* d_sub = nullptr;
    if (cudaMalloc(&d_sub, sizeof(GenzParams) * np) != cudaSuccess)
      return cuda_error(cudaErrorMemoryAllocation, "fallback params");
    std::unique_ptr<GenzParams, decltype(&cudaFree)> sub_guard(d_sub, cudaFree);
    std::vector<GenzParams> hp;
    std::vector<double> per, pea;
    std::vector<Result> pres;
    const int rc = grouped_batch(np, o, [&](const std::vector<int>& idx, Result* g) {
      const int gn = (int)idx.size();
      hp.resize(gn);
      per.assign(gn, epsrel);
      pea.assign(gn, epsabs);
      for (int j = 0; j < gn; ++j) hp[j] = h[plain_idx[idx[j]]];
      if (cudaMemcpyAsync(d_sub, hp.data(), sizeof(GenzParams) * gn, cudaMemcpyHostToDevice, s) !=
          cudaSuccess)
        return (int)kErrCuda;
      detail::ParamSource<F> gs{d_sub};
      return run_batch<kCvDim>(ws, gs, gn, per.data(), pea.data(), o, g, s);
    }, pres, &ws);
    if (rc != kOk && rc != kErrCapacity) return engine_status(ctx, rc);
    for (int j = 0; j < np; ++j) result_to_c(pres[j], &out[plain_idx[j]]);
  }
  st->ms_integrate = now_ms() - t0;
  st->mean_residual_ratio = rho_sum / count;
  return 0;
}

}  // namespace

void cub_cv_default_options(cub_cv_options* o) {
  if (!o) return;
  o->samples = 8192;
  o->batch = 1024;
  o->epochs = 30;
  o->lr = 2e-3f;
  o->rho_max = 0.5;
  o->coarse_epsrel = 1e-3;
  o->seed = 1;
}

int cub_cv_integrate_batch(cub_ctx* ctx, int family, int count, const cub_genz_params* params,
                           double epsrel, double epsabs, const cub_cv_options* opt,
                           cub_result* out, cub_cv_stats* stats) {
  if (!ctx || !params || !out || count <= 0 || !(epsrel >= 0) || !(epsabs >= 0)) {
    set_error("invalid argument");
    return CUB_ERR_INVALID;
  }
  cub_cv_options co;
  cub_cv_default_options(&co);
  if (opt) co = *opt;
  if (co.batch <= 0 || co.batch % 128 || co.samples <= 0 || co.samples % co.batch) {
    set_error("cv options: batch a multiple of 128, samples a multiple of batch");
    return CUB_ERR_INVALID;
  }
  cub_cv_stats local{};
  cub_cv_stats* st = stats ? stats : &local;
  std::memset(st, 0, sizeof(*st));
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_error(e, "cudaSetDevice");
  const GenzParams* h = reinterpret_cast<const GenzParams*>(params);
  switch (family) {
    case CUB_PRODUCT_PEAK: return cv_run<ProductPeak>(ctx, count, h, epsrel, epsabs, co, out, st);
    case CUB_GAUSSIAN: return cv_run<Gaussian>(ctx, count, h, epsrel, epsabs, co, out, st);
  }
  set_error("the control variate is built for the product-peak and Gaussian families");
  return CUB_ERR_UNSUPPORTED;
}
