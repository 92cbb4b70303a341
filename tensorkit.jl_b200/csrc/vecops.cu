// Vector-space operations on whole data vectors: y = β·y + α·x (add!, scale!;
// src/tensors/vectorinterface.jl:60-99). Two tensors of one space share their storage layout, so no
// transform table is involved: one pass over flat vectors.
//
// Bound: HBM. A thread keeps four 16-byte accesses of x (and of y when β ≠ 0) in flight; vectors
// that are not 16-byte aligned take 8-byte accesses. On 10.6 M doubles (SU(2) two-site tensor, caches cold
// at the start): β = 0 21.5 us, β = 1 32.5 us (part of the 85 MB written is still in L2 at the end: the HBM copy
// rate would take 25.9 and 38.8); as an identity permutation through the transform table 101 and 149 us.
#include <algorithm>

#include "tkb_internal.h"

namespace {

constexpr int kVecThreads = 256;
constexpr int kVecBatch = 4;  // accesses of x in flight per thread

struct CDbl {
  double x, y;
};

__device__ __forceinline__ double axpby1(double x, double y, CDbl a, CDbl b, bool bz) {
  const double r = a.x * x;
  return bz ? r : fma(b.x, y, r);
}
// a pair of real elements
struct RealOp {
  using T = double;
  static __device__ __forceinline__ double run(double x, double y, CDbl a, CDbl b, bool bz) {
    return axpby1(x, y, a, b, bz);
  }
};
struct PairOp {
  using T = double2;
  static __device__ __forceinline__ double2 run(double2 x, double2 y, CDbl a, CDbl b, bool bz) {
    return make_double2(axpby1(x.x, y.x, a, b, bz), axpby1(x.y, y.y, a, b, bz));
  }
};
struct CplxOp {
  using T = double2;
  static __device__ __forceinline__ double2 run(double2 x, double2 y, CDbl a, CDbl b, bool bz) {
    double2 r = make_double2(fma(a.x, x.x, -__dmul_rn(a.y, x.y)), fma(a.x, x.y, __dmul_rn(a.y, x.x)));
    if (!bz) {
      r.x = fma(b.x, y.x, fma(-b.y, y.y, r.x));
      r.y = fma(b.x, y.y, fma(b.y, y.x, r.y));
    }
    return r;
  }
};

// n elements of OP::T; dst may be src (every element is read before it is written, by one thread).
// odd: a single real element follows the n pairs.
template <typename OP>
__global__ void __launch_bounds__(kVecThreads)
    axpby_kernel(int64_t n, typename OP::T *dst, const typename OP::T *src, CDbl a, CDbl b, int beta_zero,
                 int odd) {
  using T = typename OP::T;
  const bool bz = beta_zero != 0;
  pdl_wait();  // both vectors belong to earlier kernels of the stream
  pdl_trigger();
  const int64_t step = (int64_t)gridDim.x * kVecThreads * kVecBatch;
  for (int64_t e0 = (int64_t)blockIdx.x * kVecThreads * kVecBatch + threadIdx.x; e0 < n; e0 += step) {
    T x[kVecBatch], y[kVecBatch];
#pragma unroll
    for (int q = 0; q < kVecBatch; ++q) {
      const int64_t e = e0 + q * kVecThreads;
      if (e < n) {
        x[q] = src[e];
        if (!bz) y[q] = dst[e];
      }
    }
#pragma unroll
    for (int q = 0; q < kVecBatch; ++q) {
      const int64_t e = e0 + q * kVecThreads;
      if (e < n) dst[e] = OP::run(x[q], y[q], a, b, bz);
    }
  }
  if (odd && blockIdx.x == 0 && threadIdx.x == 0) {
    double *d = reinterpret_cast<double *>(dst + n);
    *d = axpby1(*reinterpret_cast<const double *>(src + n), bz ? 0.0 : *d, a, b, bz);
  }
}

template <typename OP>
cudaError_t axpby_launch(tkb_ctx *ctx, int64_t n, void *dst, const void *src, CDbl a, CDbl b, int bz,
                         int odd = 0) {
  using T = typename OP::T;
  const int64_t per_cta = kVecThreads * kVecBatch;
  const int grid = (int)std::min<int64_t>(std::max<int64_t>(1, (n + per_cta - 1) / per_cta), (int64_t)ctx->num_sms * 8);
  return launch_pdl(axpby_kernel<OP>, dim3(grid), dim3(kVecThreads), 0, ctx->stream, n, (T *)dst, (const T *)src, a, b,
                    bz, odd);
}

}  // namespace

extern "C" int tkb_axpby(tkb_ctx *ctx, int dtype, int64_t n, void *dst, const void *src, tkb_scalar alpha,
                         tkb_scalar beta) {
  if (!ctx) return tkb_set_error(nullptr, TKB_ERR_ARG, "null context");
  if (dtype != TKB_F64 && dtype != TKB_C128) return tkb_set_error(ctx, TKB_ERR_ARG, "unknown dtype");
  if (n < 0) return tkb_set_error(ctx, TKB_ERR_ARG, "negative length");
  if (dtype == TKB_F64 && (alpha.im != 0.0 || beta.im != 0.0))
    return tkb_set_error(ctx, TKB_ERR_ARG, "complex scalar with real data");
  if (n == 0) return TKB_OK;
  if (!dst || !src) return tkb_set_error(ctx, TKB_ERR_ARG, "null data pointer");
  const CDbl a{alpha.re, alpha.im}, b{beta.re, beta.im};
  const int bz = (beta.re == 0.0 && beta.im == 0.0) ? 1 : 0;
  const bool aligned = (((uintptr_t)dst | (uintptr_t)src) & 15) == 0;
  if (dtype == TKB_C128) {
    if (!aligned) return tkb_set_error(ctx, TKB_ERR_ARG, "ComplexF64 data must be 16-byte aligned");
    TKB_CUDA_TRY(ctx, axpby_launch<CplxOp>(ctx, n, dst, src, a, b, bz));
  } else if (aligned) {
    TKB_CUDA_TRY(ctx, axpby_launch<PairOp>(ctx, n / 2, dst, src, a, b, bz, (int)(n & 1)));
  } else {
    TKB_CUDA_TRY(ctx, axpby_launch<RealOp>(ctx, n, dst, src, a, b, bz));
  }
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}
