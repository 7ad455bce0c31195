// mlp.cuh -- the control-variate network g: 7 -> 128 -> 128 -> 128 -> 1,
// SiLU, BF16 weights and activations, FP32 accumulation; one independent
// network per integral (batched over integrals in grid.z).
//
// Training and inference run on the tensor cores (umma.cuh: D = A * B^T with
// A, B K-major):
//
//   k_net      one CTA per 128 samples: the three hidden layers one after the
//              other, activations passed on in shared memory, weights staged
//              there once.  Inference ends with the output layer.  Training
//              goes on with the loss, the output layer's partial gradients
//              and the two backward products, and leaves H_l^T and dZ_l^T in
//              global memory.
//   k_weight_grads   dW_l = dZ_l^T H_{l-1}, one CTA per layer and network,
//              over the minibatch in a ring of asynchronous copies.
//   k_small_grads    bias and output-layer gradients, the loss.
//   k_adam     the update, and the bf16 copies of the new weights.
//
// Operands of each product:
//   forward      Z_l   = H_{l-1} W_l^T     A = H_{l-1} [s][in],  B = W_l  [out][in]
//   backward     dH_l  = dZ_{l+1} W_{l+1}  A = dZ_{l+1} [s][out], B = W^T [in][out]
//   gradients    dW_l  = dZ_l^T H_{l-1}    A = dZ_l^T [out][s],  B = H^T  [in][s]
#pragma once

#include <cuda_bf16.h>

#include "umma.cuh"

namespace cubature {
namespace mlp {

constexpr int kIn = 7;      // network inputs
constexpr int kInPad = 16;  // padded to one MMA K-step
constexpr int kHidden = 128;

__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = sigmoid(z);
  return s * (1.0f + z * (1.0f - s));
}

// Dynamic shared memory of k_gemm: the A chunk (16 KB), the B chunk (up to
// 16 KB), and slack up to 64 KB so that every operand read the descriptors
// can describe stays inside the CTA's allocation.
constexpr int kGemmSmem = 64 * 1024;

// One 128-row tile of D = A * B^T for batch entry blockIdx.z, row tile
// blockIdx.x, stored as fp32: out[e * batch_out + row * ld_out + col].
// 128 threads.
template <int N>
__global__ void __launch_bounds__(128) k_gemm(umma::GemmArgs g, float* out, long long ld_out,
                                              long long batch_out) {
  constexpr uint32_t kCols = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
  constexpr int kStep = N % 32 == 0 ? 32 : 16;
  extern __shared__ __align__(1024) uint8_t dsm[];
  uint8_t* sa = dsm;
  uint8_t* sb = dsm + umma::kTileM * umma::kChunkK * 2;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  const int e = blockIdx.z, mt = blockIdx.x;
  if (threadIdx.x == 0) umma::mbar_init(&bar, 1);
  if (threadIdx.x < 32) umma::tmem_alloc(&tmem_base, kCols);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_base;
  uint32_t phase = 0;
  const bool ok = umma::gemm_tile<N>(g, e, mt, tmem, sa, sb, &bar, phase);
  if (ok) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = mt * umma::kTileM + w * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(w * 32) << 16);
    float* o = out + (long long)e * batch_out + (long long)row * ld_out;
#pragma unroll 1
    for (int c0 = 0; c0 < N; c0 += kStep) {
      float v[kStep];
      if constexpr (kStep == 32)
        umma::tmem_load32(lane_addr + c0, v);
      else
        umma::tmem_load16(lane_addr + c0, v);
#pragma unroll
      for (int i = 0; i < kStep; ++i) o[c0 + i] = v[i];
    }
  } else {
    if (threadIdx.x == 0) atomicExch(g.error, 1);
    // the last commit may still be in flight: wait for it (bounded) before
    // the accumulator columns are released
    umma::mbar_wait(&bar, phase ^ 1);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) umma::tmem_dealloc(tmem, kCols);
}

// Layout of one network's fp32 parameter vector (also of its gradient and
// Adam moments).  W0 is [128][16] (out-major; inputs 7..15 are padding and
// stay zero), W1, W2 are [128][128] (out-major), w3 the output weights.
struct Layout {
  static constexpr int W0 = 0;
  static constexpr int B0 = W0 + kHidden * kInPad;
  static constexpr int W1 = B0 + kHidden;
  static constexpr int B1 = W1 + kHidden * kHidden;
  static constexpr int W2 = B1 + kHidden;
  static constexpr int B2 = W2 + kHidden * kHidden;
  static constexpr int W3 = B2 + kHidden;
  static constexpr int B3 = W3 + kHidden;
  static constexpr int kCount = B3 + 8;  // padded to 8 floats
};

// Inputs of network e: x in [0,1]^7 (fp64, [count][7]) -> bf16 (2x - 1),
// padded to 16, row-major X [count][16] and transposed XT [16][ld_t].
__global__ void k_prep_inputs(const double* x, long long count, long long batch_x,
                              __nv_bfloat16* X, __nv_bfloat16* XT, long long ld_t,
                              long long batch_X, long long batch_XT) {
  const int e = blockIdx.z;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < count;
       s += (long long)gridDim.x * blockDim.x) {
#pragma unroll
    for (int i = 0; i < kInPad; ++i) {
      const float v = i < kIn ? (float)(2.0 * x[e * batch_x + s * kIn + i] - 1.0) : 0.0f;
      const __nv_bfloat16 b = __float2bfloat16(v);
      X[e * batch_X + s * kInPad + i] = b;
      XT[e * batch_XT + (long long)i * ld_t + s] = b;
    }
  }
}

// Operand tiles of k_net in dynamic shared memory, each in the K-major core
// layout of umma.cuh with all of K side by side (chunk_offset of 128 rows):
// the activations (A), the inputs and the weights.
constexpr int kActBytes = 128 * 128 * 2, kInBytes = 128 * kInPad * 2;
template <bool kTrain>
constexpr int kNetSmem = kActBytes + 2 * kInBytes + (kTrain ? 4 : 2) * kActBytes;

struct NetArgs {
  const float* P;                                          // [E][Layout::kCount]
  const __nv_bfloat16 *W0, *W1, *W2, *W1T, *W2T;           // [E]
  int* error;
  // training: X row-major [E][S][16] from sample s0 on, targets, and what
  // the gradients need: H_l^T and dZ_l^T [E][128][rows], Z_1 and Z_2 by
  // sample (scratch), per-tile output-layer partials
  const __nv_bfloat16* X;
  long long batch_X;
  const float* y;
  long long batch_y;
  float inv_nbatch;
  __nv_bfloat16 *Z1, *Z2, *H1T, *H2T, *dZ1T, *dZ2T, *dZ3T;
  float* part;
  long long rows;
  // inference: x fp64 [E][n][7] -> g fp64 [E][n]
  const double* x;
  long long n;
  const float* scale;
  double* g;
};

// Copy a [rows][k] bf16 matrix (row-major, k a multiple of 8) into the core
// layout with 16-byte asynchronous copies.
__device__ __forceinline__ void stage_async(uint8_t* dst, const __nv_bfloat16* src, int rows,
                                            int k) {
  const int per = k / 8;
  for (int v = threadIdx.x; v < rows * per; v += blockDim.x) {
    const int r = v / per, c = v % per;
    umma::cp_async16(dst + umma::chunk_offset(rows, r, c * 8), src + (long long)r * k + c * 8);
  }
}

// D = A B^T of two staged operands (128 rows each, K = 16 ksteps), from one
// thread; the commit arrives on bar.
__device__ __forceinline__ void net_mma(uint32_t tmem, const uint8_t* a, const uint8_t* b,
                                        int ksteps, uint64_t* bar) {
  constexpr uint32_t idesc = umma::instr_desc_bf16(128);
  umma::fence_after_sync();
  for (int s = 0; s < ksteps; ++s) {
    const uint64_t ad = umma::smem_desc(umma::smem_u32(a) + s * 2 * (128 * 16), 128 * 16, 128);
    const uint64_t bd = umma::smem_desc(umma::smem_u32(b) + s * 2 * (128 * 16), 128 * 16, 128);
    umma::mma_bf16(tmem, ad, bd, idesc, s > 0 ? 1u : 0u);
  }
  umma::mma_commit(bar);
}

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 a, __nv_bfloat16 b) {
  return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
__device__ __forceinline__ __nv_bfloat16 unpack_bf16(uint32_t w, int hi) {
  return __ushort_as_bfloat16((unsigned short)(hi ? w >> 16 : w & 0xffffu));
}

// One 128-sample tile, 512 threads: thread t owns row t % 128 of the tile and,
// in the epilogues, 32 of its 128 columns (four warps share each quarter of
// the accumulators' lanes; with one thread per row the five epilogues were a
// chain of 128 sigmoids each and took 108 us of a step).  The
// activations go from the accumulators (TMEM) through the epilogue straight
// into the next product's A operand in shared memory, so a step is one launch
// for what took eight (and the transposes, which the weight gradients read,
// are the only activations written): 820 us a training step before, of which
// the three forward products took 3 x 78 us on scattered 2-byte stores.
// Bound now by the serial chain of five products and their epilogues.
constexpr int kNetThreads = 512;

template <bool kTrain>
__global__ void __launch_bounds__(kNetThreads) k_net(NetArgs g) {
  extern __shared__ __align__(1024) uint8_t dsm[];
  uint8_t* act = dsm;
  uint8_t* xin = act + kActBytes;
  uint8_t* w0 = xin + kInBytes;
  uint8_t* w1 = w0 + kInBytes;
  uint8_t* w2 = w1 + kActBytes;
  uint8_t* w1t = w2 + kActBytes;  // training only
  uint8_t* w2t = w1t + kActBytes;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ float bias[3][kHidden], w3[kHidden], es[kHidden], sq[kHidden];
  const int e = blockIdx.z, t = threadIdx.x;
  const int r = t & 127, c0 = (t >> 7) * 32;  // this thread's row and columns
  const float* p = g.P + (long long)e * Layout::kCount;
  stage_async(w0, g.W0 + (long long)e * kHidden * kInPad, 128, kInPad);
  stage_async(w1, g.W1 + (long long)e * kHidden * kHidden, 128, 128);
  stage_async(w2, g.W2 + (long long)e * kHidden * kHidden, 128, 128);
  if (kTrain) {
    stage_async(w1t, g.W1T + (long long)e * kHidden * kHidden, 128, 128);
    stage_async(w2t, g.W2T + (long long)e * kHidden * kHidden, 128, 128);
  }
  if (t < kHidden) {
    bias[0][t] = p[Layout::B0 + t];
    bias[1][t] = p[Layout::B1 + t];
    bias[2][t] = p[Layout::B2 + t];
    w3[t] = p[Layout::W3 + t];
  }
  const float b3 = p[Layout::B3];
  if (t == 0) umma::mbar_init(&bar, 1);
  if (t < 32) umma::tmem_alloc(&tmem_base, 128);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_base;
  const uint32_t lane_addr = tmem + ((uint32_t)((r >> 5) * 32) << 16);
  uint32_t phase = 0;
  bool ok = true;
  // one product and its wait; false (for the whole block) when it gave up
  auto product = [&](const uint8_t* a, const uint8_t* b, int ksteps) {
    umma::fence_smem_async();
    umma::fence_before_sync();
    __syncthreads();
    if (t == 0) net_mma(tmem, a, b, ksteps, &bar);
    ok = __syncthreads_and(umma::mbar_wait(&bar, phase) ? 1 : 0) != 0;
    phase ^= 1;
    umma::fence_after_sync();
    return ok;
  };
  // this thread's 32 columns into the A operand
  auto put = [&](const uint32_t (&w)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<uint4*>(act + umma::chunk_offset(128, r, c0 + 8 * i)) =
          make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  };
  const long long tiles = kTrain ? gridDim.x : (g.n + 127) / 128;
  for (long long tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
    const long long row = tile * 128 + r;
    if (kTrain) {
      stage_async(xin, g.X + (long long)e * g.batch_X + tile * 128 * kInPad, 128, kInPad);
    } else if (t < 128) {
      uint32_t w[4] = {0, 0, 0, 0};
      if (row < g.n) {
        const double* x = g.x + ((long long)e * g.n + row) * kIn;
        __nv_bfloat16 b[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          b[i] = __float2bfloat16(i < kIn ? (float)(2.0 * x[i < kIn ? i : 0] - 1.0) : 0.0f);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = pack_bf16(b[2 * i], b[2 * i + 1]);
      }
      *reinterpret_cast<uint4*>(xin + umma::chunk_offset(128, r, 0)) =
          make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(xin + umma::chunk_offset(128, r, 8)) = make_uint4(0, 0, 0, 0);
    }
    umma::cp_async_wait_all();
    const long long zrow = ((long long)e * g.rows + row) * kHidden + c0;
    const long long trow = ((long long)e * kHidden + c0) * g.rows + row;
#pragma unroll 1
    for (int l = 0; l < 3; ++l) {
      if (!product(l == 0 ? xin : act, l == 0 ? w0 : l == 1 ? w1 : w2, l == 0 ? 1 : 8)) break;
      __nv_bfloat16* Z = l == 0 ? g.Z1 : g.Z2;
      __nv_bfloat16* HT = l == 0 ? g.H1T : g.H2T;
      float v[32];
      umma::tmem_load32(lane_addr + c0, v);
      uint32_t zw[16], hw[16];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        __nv_bfloat16 zb[2], hb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          zb[u] = __float2bfloat16(v[i + u] + bias[l][c0 + i + u]);
          hb[u] = __float2bfloat16(silu(__bfloat162float(zb[u])));
          if (kTrain && l < 2) HT[trow + (long long)(i + u) * g.rows] = hb[u];
        }
        zw[i / 2] = pack_bf16(zb[0], zb[1]);
        hw[i / 2] = pack_bf16(hb[0], hb[1]);
      }
      put(hw);
      if (kTrain && l < 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(Z + zrow + 8 * i) =
              make_uint4(zw[4 * i], zw[4 * i + 1], zw[4 * i + 2], zw[4 * i + 3]);
      }
    }
    if (!ok) break;
    __syncthreads();
    // the output layer, a thread per row, columns in order
    if (t < 128) {
      float out = b3;
#pragma unroll 4
      for (int c = 0; c < 128; c += 8) {
        const uint4 q = *reinterpret_cast<const uint4*>(act + umma::chunk_offset(128, r, c));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 8; ++i)
          out += __bfloat162float(unpack_bf16(w[i / 2], i & 1)) * w3[c + i];
      }
      if constexpr (!kTrain) {
        if (row < g.n) g.g[(long long)e * g.n + row] = (double)g.scale[e] * (double)out;
      } else {
        // loss: err = g - y, e = 2 err / nbatch
        const float err = out - g.y[(long long)e * g.batch_y + row];
        es[t] = 2.0f * err * g.inv_nbatch;
        sq[t] = err * err;
      }
    }
    if constexpr (kTrain) {
      __syncthreads();
      // this tile's partial sums (fixed order): sum_s e H3[s][:] by the first
      // 128 threads, sum_s e and sum_s err^2 by another warp's first thread
      float* po = g.part + ((long long)e * gridDim.x + blockIdx.x) * (kHidden + 2);
      if (t < 128) {
        float acc = 0;
#pragma unroll 8
        for (int i = 0; i < 128; ++i)
          acc += es[i] * __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(
                             act + umma::chunk_offset(128, i, t)));
        po[t] = acc;
      } else if (t == 128) {
        float se = 0, ss = 0;
#pragma unroll 8
        for (int i = 0; i < 128; ++i) {
          se += es[i];
          ss += sq[i];
        }
        po[kHidden] = se;
        po[kHidden + 1] = ss;
      }
      const float ec = es[r];
      __syncthreads();  // H3 is read; its tile becomes dZ3
#pragma unroll 1
      for (int l = 2; l >= 0; --l) {
        // dZ_3 = e w3 silu'(Z_3) from the third product's accumulators, then
        // dZ_l = dH_l silu'(Z_l)
        if (l < 2 && !product(act, l == 1 ? w2t : w1t, 8)) break;
        __nv_bfloat16* T = l == 2 ? g.dZ3T : l == 1 ? g.dZ2T : g.dZ1T;
        const __nv_bfloat16* Z = l == 1 ? g.Z2 : g.Z1;
        uint32_t zw[16], dw[16];
        if (l < 2) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 q = *reinterpret_cast<const uint4*>(Z + zrow + 8 * i);
            zw[4 * i] = q.x;
            zw[4 * i + 1] = q.y;
            zw[4 * i + 2] = q.z;
            zw[4 * i + 3] = q.w;
          }
        }
        float v[32];
        umma::tmem_load32(lane_addr + c0, v);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          __nv_bfloat16 db[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float dz;
            if (l == 2) {
              const __nv_bfloat16 zb = __float2bfloat16(v[i + u] + bias[2][c0 + i + u]);
              dz = ec * w3[c0 + i + u] * silu_grad(__bfloat162float(zb));
            } else {
              dz = v[i + u] * silu_grad(__bfloat162float(unpack_bf16(zw[i / 2], u)));
            }
            db[u] = __float2bfloat16(dz);
            T[trow + (long long)(i + u) * g.rows] = db[u];
          }
          dw[i / 2] = pack_bf16(db[0], db[1]);
        }
        if (l > 0) put(dw);
      }
    }
  }
  if (!ok) {
    if (t == 0) atomicExch(g.error, 1);
    // the last commit may still be in flight: wait for it (bounded) before
    // the accumulator columns and the operands are released
    umma::mbar_wait(&bar, phase ^ 1);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (t < 32) umma::tmem_dealloc(tmem, 128);
}

// Weight gradients of network blockIdx.z, layer blockIdx.x (0, 1, 2):
// dW_l = dZ_l^T H_{l-1} over the minibatch, K in chunks of 64 samples through
// a ring of kGradStages chunks filled by asynchronous copies (the serial
// copy, wait, multiply of one chunk took 8.6 us, 138 us for a minibatch of
// 1024).
constexpr int kGradStages = 4;
constexpr int kGradStageBytes = 2 * umma::kTileM * umma::kChunkK * 2;
constexpr int kGradSmem = kGradStages * kGradStageBytes;

struct GradArgs {
  const __nv_bfloat16 *dZT[3];  // [E][128][rows]
  const __nv_bfloat16 *HT[3];   // layer 0: XT [E][16][ldx] from sample s0 on
  long long ldx, rows;
  float* G;  // [E][Layout::kCount]
  int* error;
};

__global__ void __launch_bounds__(128) k_weight_grads(GradArgs g) {
  extern __shared__ __align__(1024) uint8_t dsm[];
  __shared__ uint64_t bar[kGradStages];
  __shared__ uint32_t tmem_base;
  const int l = blockIdx.x, e = blockIdx.z, t = threadIdx.x;
  const int n = l == 0 ? kInPad : kHidden;  // rows of B
  const __nv_bfloat16* A = g.dZT[l] + (long long)e * kHidden * g.rows;
  const long long ldb = l == 0 ? g.ldx : g.rows;
  const __nv_bfloat16* B = g.HT[l] + (long long)e * n * ldb;
  const int nc = (int)(g.rows / umma::kChunkK);
  if (t < kGradStages) umma::mbar_init(&bar[t], 1);
  if (t < 32) umma::tmem_alloc(&tmem_base, 128);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = umma::instr_desc_bf16(n);
  auto load = [&](int c) {
    uint8_t* sa = dsm + (c % kGradStages) * kGradStageBytes;
    uint8_t* sb = sa + umma::kTileM * umma::kChunkK * 2;
    const long long k0 = (long long)c * umma::kChunkK;
    for (int v = t; v < umma::kTileM * 8; v += 128)
      umma::cp_async16(sa + umma::chunk_offset(umma::kTileM, v / 8, v % 8 * 8),
                       A + (long long)(v / 8) * g.rows + k0 + v % 8 * 8);
    for (int v = t; v < n * 8; v += 128)
      umma::cp_async16(sb + umma::chunk_offset(n, v / 8, v % 8 * 8),
                       B + (long long)(v / 8) * ldb + k0 + v % 8 * 8);
  };
  for (int c = 0; c < kGradStages - 1; ++c) {
    if (c < nc) load(c);
    umma::cp_async_commit();
  }
  bool ok = true, good = true;  // the block's verdict, this thread's waits
  int issued = 0;               // products committed
  for (int c = 0; c < nc; ++c) {
    umma::cp_async_wait<kGradStages - 2>();
    umma::fence_smem_async();
    ok = __syncthreads_and(good ? 1 : 0) != 0;
    if (!ok) break;
    if (t == 0) {
      umma::fence_after_sync();
      const uint32_t sa = umma::smem_u32(dsm + (c % kGradStages) * kGradStageBytes);
      const uint32_t sb = sa + umma::kTileM * umma::kChunkK * 2;
      for (int s = 0; s < umma::kChunkK / 16; ++s)
        umma::mma_bf16(tmem,
                       umma::smem_desc(sa + s * 2 * (umma::kTileM * 16), umma::kTileM * 16, 128),
                       umma::smem_desc(sb + s * 2 * (n * 16), n * 16, 128), idesc,
                       c > 0 || s > 0 ? 1u : 0u);
      umma::mma_commit(&bar[c % kGradStages]);
    }
    ++issued;
    // the stage that chunk c + 3 goes to is free when product c - 1 is done
    if (c >= 1)
      good = umma::mbar_wait(&bar[(c - 1) % kGradStages], (uint32_t)((c - 1) / kGradStages) & 1u);
    if (good && c + kGradStages - 1 < nc) load(c + kGradStages - 1);
    umma::cp_async_commit();
  }
  umma::cp_async_wait_all();
  // every product's end (bounded waits), also after one gave up
  if (issued > 0) {
    const int c = issued - 1;
    good = umma::mbar_wait(&bar[c % kGradStages], (uint32_t)(c / kGradStages) & 1u) && good;
    ok = __syncthreads_and(good ? 1 : 0) != 0 && ok;
  }
  umma::fence_after_sync();
  if (ok) {
    const uint32_t lane_addr = tmem + ((uint32_t)((t >> 5) * 32) << 16);
    float* o = g.G + (long long)e * Layout::kCount +
               (l == 0 ? Layout::W0 : l == 1 ? Layout::W1 : Layout::W2) + (long long)t * n;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += 16) {
      float v[16];
      umma::tmem_load16(lane_addr + c0, v);
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        *reinterpret_cast<float4*>(o + c0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
  } else if (t == 0) {
    atomicExch(g.error, 1);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (t < 32) umma::tmem_dealloc(tmem, 128);
}

// Bias gradients, a warp per hidden unit: G[b_l + j] = sum_s dZ_l^T[j][s]
// (blocks 0 .. 47, layer blockIdx.x / 16; lane-strided, then a shuffle tree),
// and in block 48 the output layer's gradients and the loss: the per-tile
// partials summed in tile order.
__global__ void __launch_bounds__(256) k_small_grads(GradArgs g, const float* part, int ntiles,
                                                     float* loss, float inv_nbatch) {
  const int e = blockIdx.z;
  float* G = g.G + (long long)e * Layout::kCount;
  if (blockIdx.x < 48) {
    const int l = blockIdx.x / 16, j = (blockIdx.x % 16) * 8 + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* r = g.dZT[l] + ((long long)e * kHidden + j) * g.rows;
    float a = 0;
    for (long long s = lane; s < g.rows; s += 32) a += __bfloat162float(r[s]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) G[(l == 0 ? Layout::B0 : l == 1 ? Layout::B1 : Layout::B2) + j] = a;
    return;
  }
  const float* pe = part + (long long)e * ntiles * (kHidden + 2);
  for (int j = threadIdx.x; j < kHidden + 2; j += blockDim.x) {
    float a = 0;
    for (int b = 0; b < ntiles; ++b) a += pe[(long long)b * (kHidden + 2) + j];
    if (j < kHidden)
      G[Layout::W3 + j] = a;
    else if (j == kHidden)
      G[Layout::B3] = a;
    else
      loss[e] = a * inv_nbatch;
  }
}

// bf16 copies of weight i (index in a network's parameters) for the tensor
// cores: W0, W1, W2 (out-major) and W1T, W2T (in-major).
struct BfWeights {
  __nv_bfloat16 *W0, *W1, *W1T, *W2, *W2T;
  __device__ __forceinline__ void put(int e, int i, float v) const {
    const __nv_bfloat16 b = __float2bfloat16(v);
    const long long sq = (long long)e * kHidden * kHidden;
    if (i < Layout::B0) {
      W0[(long long)e * kHidden * kInPad + i] = b;
    } else if (i >= Layout::W1 && i < Layout::B1) {
      const int q = i - Layout::W1;
      W1[sq + q] = b;
      W1T[sq + (q % kHidden) * kHidden + q / kHidden] = b;
    } else if (i >= Layout::W2 && i < Layout::B2) {
      const int q = i - Layout::W2;
      W2[sq + q] = b;
      W2T[sq + (q % kHidden) * kHidden + q / kHidden] = b;
    }
  }
};

// Adam on every parameter of every network (step t >= 1, bias-corrected),
// and the tensor cores' copies of the new weights.
__global__ void k_adam(float* P, const float* G, float* M, float* V, long long n, float lr,
                       float b1, float b2, float eps, float c1, float c2, BfWeights w) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float g = G[i];
    const float m = b1 * M[i] + (1 - b1) * g;
    const float v = b2 * V[i] + (1 - b2) * g * g;
    M[i] = m;
    V[i] = v;
    P[i] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
    w.put((int)(i / Layout::kCount), (int)(i % Layout::kCount), P[i]);
  }
}

// The copies alone (parameters set from the host).
__global__ void k_refresh_weights(const float* P, long long n, BfWeights w) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    w.put((int)(i / Layout::kCount), (int)(i % Layout::kCount), P[i]);
}

// Starting parameters: the draws of a 64-bit LCG (x -> kLcgA x + kLcgC from x0,
// the uniform value in the high 53 bits), in the order of networks, then W0
// (seven of sixteen columns), W1, W2, w3; uniform in +-1/sqrt(fan in), zero
// biases and padding.  A thread jumps to its first draw (repeated squaring of
// the step) and walks kInitRun of them: the host took 80 us a network for the
// same serial sequence.
constexpr unsigned long long kLcgA = 6364136223846793005ull, kLcgC = 1442695040888963407ull;
constexpr int kInitDraws = kHidden * kIn + 2 * kHidden * kHidden + kHidden;  // per network
constexpr int kInitRun = 32;

__global__ void k_init_params(float* P, int count, unsigned long long x0) {
  const long long total = (long long)count * kInitDraws;
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kInitRun;
  if (first >= total) return;
  // x0 after `first` steps
  unsigned long long a = kLcgA, c = kLcgC, x = x0;
  for (unsigned long long n = (unsigned long long)first; n; n >>= 1) {
    if (n & 1) x = a * x + c;
    c = (a + 1) * c;
    a = a * a;
  }
  const double a0 = 1.0 / sqrt((double)kIn), ah = 1.0 / sqrt(128.0);
  for (long long d = first; d < first + kInitRun && d < total; ++d) {
    x = kLcgA * x + kLcgC;
    const double u = (double)(x >> 11) * (1.0 / 9007199254740992.0);
    int i = (int)(d % kInitDraws), at;
    const bool in = i < kHidden * kIn;
    if (in) {
      at = Layout::W0 + i / kIn * kInPad + i % kIn;
    } else if ((i -= kHidden * kIn) < kHidden * kHidden) {
      at = Layout::W1 + i;
    } else if ((i -= kHidden * kHidden) < kHidden * kHidden) {
      at = Layout::W2 + i;
    } else {
      at = Layout::W3 + i - kHidden * kHidden;
    }
    P[d / kInitDraws * Layout::kCount + at] = (float)((2 * u - 1) * (in ? a0 : ah));
  }
}

// Targets of network e scaled by 1 / max |y| (scale[e] = max |y|, 1 if 0).
__global__ void k_scale_targets(const double* y, long long count, float* Y, float* scale) {
  const int e = blockIdx.z;
  __shared__ double red[256];
  double m = 0;
  for (long long s = threadIdx.x; s < count; s += blockDim.x) m = fmax(m, fabs(y[e * count + s]));
  red[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
    __syncthreads();
  }
  const double sc = red[0] > 0 ? red[0] : 1.0;
  if (threadIdx.x == 0) scale[e] = (float)sc;
  for (long long s = threadIdx.x; s < count; s += blockDim.x)
    Y[e * count + s] = (float)(y[e * count + s] / sc);
}

}  // namespace mlp
}  // namespace cubature
