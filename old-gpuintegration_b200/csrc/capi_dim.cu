// capi_dim.cu -- instantiations of the engine for one dimension, compiled
// once per dimension and family (-DCUB_DIM=N -DCUB_FAMILY=Gaussian, ...: the
// family's kernels), and once per dimension without a family (dispatch over
// the families, mixed batches, the split step).  A unit per family keeps the
// units small enough to compile side by side.
#include "capi_internal.h"
#include "cubature/step_kernels.cuh"

#ifndef CUB_DIM
#error "compile with -DCUB_DIM=<ndim>"
#endif

#define CUB_CAT2(a, b) a##b
#define CUB_CAT(a, b) CUB_CAT2(a, b)

namespace cubature {
namespace capi {

// What a family provides in N dimensions.
template <int N, template <int> class Fam>
struct FamilyDim {
  static int run(cub_ctx* ctx, int count, const GenzParams* h_params, const GenzParams* d_params,
                 const double* epsrel, const double* epsabs, const Options& opt, Result* out,
                 const double* h_box);
  static int rule(const GenzParams& p, long long n, const double* lo, const double* len,
                  long long ld, double epsrel, double epsabs, double* avg, double* err, int* axis,
                  int* active, cudaStream_t s);
  // A batch of the family for replay: its integrands read their parameters
  // from device memory, so one recording serves every call.
  static int replay_prepare(Workspace& ws, int count, const Options& opt, cudaStream_t s,
                            Replay* r);
  static int replay_enqueue(Workspace& ws, const GenzParams* d_params, const Replay& r,
                            cudaStream_t s);
};

#ifdef CUB_FAMILY

template <int N, template <int> class Fam>
int FamilyDim<N, Fam>::run(cub_ctx* ctx, int count, const GenzParams* h_params,
                           const GenzParams* d_params, const double* epsrel,
                           const double* epsabs, const Options& opt, Result* out,
                           const double* h_box) {
  if (count == 1) {
    detail::SingleSource<Fam<N>> src{Fam<N>::load(h_params[0])};
    return run_batch<N>(*ctx->ws, src, 1, epsrel, epsabs, opt, out, ctx->stream, h_box);
  }
  detail::ParamSource<Fam<N>> src{d_params};
  return run_batch<N>(*ctx->ws, src, count, epsrel, epsabs, opt, out, ctx->stream, h_box);
}

template <int N, template <int> class Fam>
int FamilyDim<N, Fam>::rule(const GenzParams& p, long long n, const double* lo, const double* len,
                            long long ld, double epsrel, double epsabs, double* avg, double* err,
                            int* axis, int* active, cudaStream_t s) {
  const RuleTables T = make_rule9_tables(N);
  const Fam<N> f = Fam<N>::load(p);
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = sm_count(dev);
  if (n >= rule_thread_min<Fam<N>>(sms)) {
    constexpr int kThreads = detail::kFactored<Fam<N>> ? 128 : 256;
    const long long blocks =
        std::min<long long>((n + kThreads - 1) / kThreads, (long long)sms * 32);
    k_step_rule<N, 1><<<(unsigned)blocks, kThreads, 0, s>>>(f, T, n, lo, len, ld, epsrel, epsabs,
                                                            avg, err, axis, active);
  } else {
    const long long blocks = std::max<long long>(1, (n * 32 + 255) / 256);
    k_step_rule<N, 32><<<(unsigned)std::min<long long>(blocks, (long long)sms * 32), 256, 0, s>>>(
        f, T, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active);
  }
  return 0;
}

template <int N, template <int> class Fam>
int FamilyDim<N, Fam>::replay_prepare(Workspace& ws, int count, const Options& opt,
                                      cudaStream_t s, Replay* r) {
  return cubature::replay_prepare<N, detail::ParamSource<Fam<N>>>(ws, count, opt, s, r);
}

template <int N, template <int> class Fam>
int FamilyDim<N, Fam>::replay_enqueue(Workspace& ws, const GenzParams* d_params, const Replay& r,
                                      cudaStream_t s) {
  return cubature::replay_enqueue<N>(ws, detail::ParamSource<Fam<N>>{d_params}, r, s);
}

template struct FamilyDim<CUB_DIM, CUB_FAMILY>;

#else

namespace {
constexpr int N = CUB_DIM;
}

int CUB_CAT(replay_prepare_dim_, CUB_DIM)(int family, Workspace& ws, int count,
                                          const Options& opt, cudaStream_t s, Replay* r) {
  switch (family) {
    case kGaussian: return FamilyDim<N, Gaussian>::replay_prepare(ws, count, opt, s, r);
    case kOscillatory: return FamilyDim<N, Oscillatory>::replay_prepare(ws, count, opt, s, r);
    case kCornerPeak: return FamilyDim<N, CornerPeak>::replay_prepare(ws, count, opt, s, r);
    case kProductPeak: return FamilyDim<N, ProductPeak>::replay_prepare(ws, count, opt, s, r);
    case kContinuous: return FamilyDim<N, Continuous>::replay_prepare(ws, count, opt, s, r);
    case kDiscontinuous: return FamilyDim<N, Discontinuous>::replay_prepare(ws, count, opt, s, r);
    case kCosSum: return FamilyDim<N, CosSum>::replay_prepare(ws, count, opt, s, r);
  }
  return CUB_ERR_INVALID;
}

int CUB_CAT(replay_enqueue_dim_, CUB_DIM)(int family, Workspace& ws, const GenzParams* d_params,
                                          const Replay& r, cudaStream_t s) {
  switch (family) {
    case kGaussian: return FamilyDim<N, Gaussian>::replay_enqueue(ws, d_params, r, s);
    case kOscillatory: return FamilyDim<N, Oscillatory>::replay_enqueue(ws, d_params, r, s);
    case kCornerPeak: return FamilyDim<N, CornerPeak>::replay_enqueue(ws, d_params, r, s);
    case kProductPeak: return FamilyDim<N, ProductPeak>::replay_enqueue(ws, d_params, r, s);
    case kContinuous: return FamilyDim<N, Continuous>::replay_enqueue(ws, d_params, r, s);
    case kDiscontinuous: return FamilyDim<N, Discontinuous>::replay_enqueue(ws, d_params, r, s);
    case kCosSum: return FamilyDim<N, CosSum>::replay_enqueue(ws, d_params, r, s);
  }
  return CUB_ERR_INVALID;
}

int CUB_CAT(run_mixed_dim_, CUB_DIM)(cub_ctx* ctx, int count, const GenzParams* d_params,
                                     const int* d_fams, const double* epsrel,
                                     const double* epsabs, const Options& opt, Result* out) {
  detail::MixedSource<N> src{d_params, d_fams};
  return run_batch<N>(*ctx->ws, src, count, epsrel, epsabs, opt, out, ctx->stream);
}

int CUB_CAT(run_dim_, CUB_DIM)(cub_ctx* ctx, int family, int count, const GenzParams* h_params,
                               const GenzParams* d_params, const double* epsrel,
                               const double* epsabs, const Options& opt, Result* out,
                               const double* h_box) {
  switch (family) {
    case kGaussian: return FamilyDim<N, Gaussian>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kOscillatory: return FamilyDim<N, Oscillatory>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kCornerPeak: return FamilyDim<N, CornerPeak>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kProductPeak: return FamilyDim<N, ProductPeak>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kContinuous: return FamilyDim<N, Continuous>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kDiscontinuous: return FamilyDim<N, Discontinuous>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
    case kCosSum: return FamilyDim<N, CosSum>::run(ctx, count, h_params, d_params, epsrel, epsabs, opt, out, h_box);
  }
  return CUB_ERR_INVALID;
}

int CUB_CAT(rule_eval_dim_, CUB_DIM)(int family, const GenzParams& p, long long n,
                                     const double* lo, const double* len, long long ld,
                                     double epsrel, double epsabs, double* avg, double* err,
                                     int* axis, int* active, cudaStream_t s) {
  switch (family) {
    case kGaussian: return FamilyDim<N, Gaussian>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kOscillatory: return FamilyDim<N, Oscillatory>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kCornerPeak: return FamilyDim<N, CornerPeak>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kProductPeak: return FamilyDim<N, ProductPeak>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kContinuous: return FamilyDim<N, Continuous>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kDiscontinuous: return FamilyDim<N, Discontinuous>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
    case kCosSum: return FamilyDim<N, CosSum>::rule(p, n, lo, len, ld, epsrel, epsabs, avg, err, axis, active, s);
  }
  return CUB_ERR_INVALID;
}

int CUB_CAT(split_dim_, CUB_DIM)(long long n, const double* lo, const double* len, long long ld,
                                 const int* active, const int* axis, double* olo, double* olen,
                                 long long old, int layout, long long* count, int* cnt,
                                 int* excl, cudaStream_t s) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = sm_count(dev);
  const long long nchunk = (n + 31) / 32;
  const unsigned blocks =
      (unsigned)std::max<long long>(1, std::min<long long>((nchunk + 7) / 8, (long long)sms * 16));
  k_step_count<<<blocks, 256, 0, s>>>(n, active, cnt);
  k_step_scan<<<1, 1024, 0, s>>>(nchunk, cnt, excl, count);
  k_step_write<N><<<blocks, 256, 0, s>>>(n, lo, len, ld, active, axis, excl, count, olo, olen,
                                         old, layout);
  return 0;
}

#endif  // CUB_FAMILY

}  // namespace capi
}  // namespace cubature
