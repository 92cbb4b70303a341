// Partial-trace transform: every destination sub-block of a trace_permute! in one launch.
//
// Semantics (TensorKit _trace_permute!, src/tensors/tensoroperations.jl:246-296, bosonic):
//   dst_g = β·dst_g + α·Σ_e coeff_e · tensortrace(src_e, p, q)      for every group g
// where the entries e of group g are the source sub-blocks whose permuted tree pairs split
// into destination pair g. The host flattens the recoupling (permute of the fusion blocks to
// ((p₁, q₁), (p₂, q₂)), split, dim ratio) into coefficients; a traced leg pair becomes one
// summation index with stride stride(q₁) + stride(q₂).
//
// Work decomposition: a task is up to `lanes` consecutive elements of one group (the destination's
// first dim is its fastest, so loads and stores coalesce), and the CTA's threads share the sums
// of each element: the group's terms (every traced position of every entry) are cut into pieces,
// thread (slice, lane) adds every slices-th piece of its element, and the slices are added pairwise
// in shared memory. The host picks lanes per group: 32, fewer where the group has fewer elements (a
// full trace has one), more where it has fewer terms than the eight slices that 32 lanes leave.
//
// Bound: latency (a trace reads few bytes: sums of tens to hundreds of scattered terms per element).
// One thread per element that walked its terms one by one took 52 us for the SU(2) trace of two
// 10 - 90 dimensional legs (1 M terms, cold caches); eight slices with eight loads in flight each
// take 13.7 us.
#include <algorithm>
#include <cstring>

#include "tkb_internal.h"

namespace {

constexpr int kTrThreads = 256;
constexpr int kTrLanes = 32;  // elements per task: whole sectors on both sides
constexpr int kTrBatch = 8;   // loads in flight per thread

struct CDbl {
  double x, y;
};

__device__ __forceinline__ double ld_src(const double *p, bool) { return __ldg(p); }
__device__ __forceinline__ double2 ld_src(const double2 *p, bool conj) {
  double2 v = __ldg(p);
  if (conj) v.y = -v.y;
  return v;
}
__device__ __forceinline__ double zero_v(double) { return 0.0; }
__device__ __forceinline__ double2 zero_v(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double add_v(double a, double b) { return a + b; }
__device__ __forceinline__ double2 add_v(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double axpy_v(double u, double v, double acc) { return fma(u, v, acc); }
__device__ __forceinline__ double2 axpy_v(double u, double2 v, double2 acc) {
  return make_double2(fma(u, v.x, acc.x), fma(u, v.y, acc.y));
}
__device__ __forceinline__ double finish_v(double v, CDbl a, CDbl b, const double *d, bool bz) {
  double r = a.x * v;
  if (!bz) r = fma(b.x, *d, r);
  return r;
}
__device__ __forceinline__ double2 finish_v(double2 v, CDbl a, CDbl b, const double2 *d, bool bz) {
  double2 r = make_double2(a.x * v.x - a.y * v.y, a.x * v.y + a.y * v.x);
  if (!bz) {
    const double2 o = *d;
    r.x = fma(b.x, o.x, fma(-b.y, o.y, r.x));
    r.y = fma(b.x, o.y, fma(b.y, o.x, r.y));
  }
  return r;
}

// NF: most free dims; MULTI: more than one traced pair (the traced multi-index of a position is
// formed by division)
template <typename T, bool CONJ, int NF, bool MULTI>
__global__ void __launch_bounds__(kTrThreads)
    trace_kernel(const TrGroup *__restrict__ groups, const TrEntry *__restrict__ entries,
                 const TrPiece *__restrict__ pieces, const int32_t *__restrict__ task_group, int64_t ntasks, int nfree,
                 int ntrace, T *__restrict__ dst, const T *__restrict__ src, CDbl alpha, CDbl beta, int beta_zero) {
  __shared__ T red[kTrThreads];
  const bool bz = beta_zero != 0;
  pdl_wait();  // source and destination belong to earlier kernels
  pdl_trigger();
  for (int64_t task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const TrGroup &G = groups[task_group[task]];
    const int lanes = G.lanes, slices = kTrThreads / lanes;
    const int lane = threadIdx.x & (lanes - 1), slice = threadIdx.x / lanes;
    const int64_t e = (task - G.task_begin) * lanes + lane;
    const bool in = e < G.nelem;
    T acc = zero_v(T{});
    int64_t doff = G.dst_off;
    if (in) {
      // free multi-index (first dim fastest)
      int32_t x[NF];
      int64_t r = e;
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        if (k < nfree) {
          const int64_t q = r <= UINT32_MAX ? (int64_t)((uint32_t)r / (uint32_t)G.size[k]) : r / G.size[k];
          x[k] = (int32_t)(r - q * G.size[k]);
          r = q;
          doff += (int64_t)x[k] * G.dstr[k];
        } else {
          x[k] = 0;
        }
      }
      for (int64_t p = G.p_begin + slice; p < G.p_end; p += slices) {
        const TrPiece P = pieces[p];
        const TrEntry &E = entries[P.entry];
        int64_t base = E.src_off;
#pragma unroll
        for (int k = 0; k < NF; ++k)
          if (k < nfree) base += (int64_t)x[k] * E.sstr[k];
        T s = zero_v(T{});
        for (int64_t t0 = 0; t0 < P.n; t0 += kTrBatch) {
          T v[kTrBatch];
#pragma unroll
          for (int q = 0; q < kTrBatch; ++q) {
            int64_t t = P.t0 + t0 + q, off = base;
            if (t0 + q < P.n) {
              if constexpr (MULTI) {
                for (int l = 0; l < ntrace; ++l) {
                  const int64_t d = t / E.tsize[l];
                  off += (t - d * E.tsize[l]) * E.tstr[l];
                  t = d;
                }
              } else {
                off += t * E.tstr[0];
              }
              v[q] = ld_src(src + off, CONJ);
            } else {
              v[q] = zero_v(T{});
            }
          }
#pragma unroll
          for (int q = 0; q < kTrBatch; ++q) s = add_v(s, v[q]);
        }
        acc = axpy_v(E.coeff, s, acc);
      }
    }
    if (slices > 1) {
      red[threadIdx.x] = acc;
      for (int h = slices / 2; h > 0; h >>= 1) {
        __syncthreads();
        if (slice < h) red[threadIdx.x] = add_v(red[threadIdx.x], red[threadIdx.x + h * lanes]);
      }
      acc = red[threadIdx.x];
      __syncthreads();  // read before the next task writes
    }
    if (in && slice == 0) {
      T *dp = dst + doff;
      *dp = finish_v(acc, alpha, beta, dp, bz);
    }
  }
}

}  // namespace

extern "C" int tkb_trace_table_create(tkb_ctx *ctx, const tkb_trace_desc *d, tkb_trace_table **out) {
  if (!ctx || !d || !out) return TKB_ERR_ARG;
  *out = nullptr;
  const int nf = d->nfree, nt = d->ntrace;
  if (nf < 0 || nf > TKB_MAX_IND || nt < 1 || nt > TKB_MAX_IND)
    return tkb_set_error(ctx, TKB_ERR_ARG, "nfree/ntrace out of range");
  const int64_t G = d->ngroups;
  if (G < 0) return tkb_set_error(ctx, TKB_ERR_ARG, "negative ngroups");
  if (G > 0 && (!d->group_entry_ptr || !d->dst_offsets || (nf > 0 && (!d->sizes || !d->dst_strides))))
    return tkb_set_error(ctx, TKB_ERR_ARG, "null group array");
  const int64_t NE = G > 0 ? d->group_entry_ptr[G] : 0;
  if (NE > 0 && (!d->src_offsets || !d->coeffs || !d->trace_sizes || !d->trace_strides ||
                 (nf > 0 && !d->src_strides)))
    return tkb_set_error(ctx, TKB_ERR_ARG, "null entry array");
  std::vector<TrGroup> hg(G);
  std::vector<TrEntry> he(NE);
  std::vector<TrPiece> hp;
  std::vector<int32_t> htask;
  int64_t ntasks = 0;
  for (int64_t g = 0; g < G; ++g) {
    TrGroup &tg = hg[g];
    std::memset(&tg, 0, sizeof(tg));
    const int64_t e0 = d->group_entry_ptr[g], e1 = d->group_entry_ptr[g + 1];
    if (e0 < 0 || e1 < e0 || e1 > NE) return tkb_set_error(ctx, TKB_ERR_ARG, "inconsistent entry pointers");
    tg.dst_off = d->dst_offsets[g];
    int64_t hi = tg.dst_off, vol = 1;
    if (hi < 0) return tkb_set_error(ctx, TKB_ERR_SIZE, "negative destination offset");
    for (int k = 0; k < nf; ++k) {
      const int64_t sz = d->sizes[g * nf + k], st = d->dst_strides[g * nf + k];
      if (sz <= 0 || sz > INT32_MAX) return tkb_set_error(ctx, TKB_ERR_SIZE, "bad free size");
      if (st < 0) return tkb_set_error(ctx, TKB_ERR_SIZE, "negative destination stride");
      tg.size[k] = (int32_t)sz;
      tg.dstr[k] = st;
      hi += (sz - 1) * st;
      vol *= sz;
    }
    if (hi >= d->dst_len)
      return tkb_set_error(ctx, TKB_ERR_SIZE, "destination sub-block exceeds its data vector");
    tg.nelem = vol;
    int64_t terms = 0;  // of one element
    for (int64_t e = e0; e < e1; ++e) {
      TrEntry &te = he[e];
      std::memset(&te, 0, sizeof(te));
      te.src_off = d->src_offsets[e];
      te.coeff = d->coeffs[e];
      int64_t shi = te.src_off, ntot = 1;
      if (shi < 0) return tkb_set_error(ctx, TKB_ERR_SIZE, "negative source offset");
      for (int k = 0; k < nf; ++k) {
        const int64_t st = d->src_strides[e * nf + k];
        if (st < 0) return tkb_set_error(ctx, TKB_ERR_SIZE, "negative source stride");
        te.sstr[k] = st;
        shi += (tg.size[k] - 1) * st;
      }
      for (int l = 0; l < nt; ++l) {
        const int64_t sz = d->trace_sizes[e * nt + l], st = d->trace_strides[e * nt + l];
        if (sz <= 0 || sz > INT32_MAX || st < 0)
          return tkb_set_error(ctx, TKB_ERR_SIZE, "bad traced size or stride");
        te.tsize[l] = (int32_t)sz;
        te.tstr[l] = st;
        shi += (sz - 1) * st;
        ntot *= sz;
      }
      te.ntr_total = ntot;
      terms += ntot;
      if (shi >= d->src_len)
        return tkb_set_error(ctx, TKB_ERR_SIZE, "source sub-block exceeds its data vector");
    }
    int lanes = 1;
    while (lanes < kTrLanes && lanes < vol) lanes <<= 1;
    while (lanes < kTrThreads && kTrThreads / lanes / 2 >= terms) lanes <<= 1;  // slices without a term
    tg.lanes = lanes;
    // pieces: about two per slice at least, equal parts of each entry
    const int64_t most = std::max<int64_t>(1, terms / (2 * (kTrThreads / lanes)));
    tg.p_begin = (int64_t)hp.size();
    for (int64_t e = e0; e < e1; ++e) {
      const int64_t ntot = he[e].ntr_total, parts = (ntot + most - 1) / most;
      for (int64_t q = 0; q < parts; ++q) {
        const int64_t a = ntot / parts * q + std::min(q, ntot % parts);
        hp.push_back({a, ntot / parts + (q < ntot % parts ? 1 : 0), e});
      }
    }
    tg.p_end = (int64_t)hp.size();
    tg.task_begin = ntasks;
    const int64_t nt_g = (vol + lanes - 1) / lanes;
    htask.insert(htask.end(), (size_t)nt_g, (int32_t)g);
    ntasks += nt_g;
  }
  tkb_trace_table *t = new tkb_trace_table();
  t->owner = ctx;
  t->nfree = nf;
  t->ntrace = nt;
  t->ngroups = G;
  t->ntasks = ntasks;
  t->src_len = d->src_len;
  t->dst_len = d->dst_len;
  auto up = [&](void **dptr, const void *h, size_t bytes) -> cudaError_t {
    if (bytes == 0) return cudaSuccess;
    cudaError_t e = cudaMalloc(dptr, bytes);
    if (e != cudaSuccess) return e;
    return cudaMemcpy(*dptr, h, bytes, cudaMemcpyHostToDevice);
  };
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e == cudaSuccess) e = up((void **)&t->groups, hg.data(), hg.size() * sizeof(TrGroup));
  if (e == cudaSuccess) e = up((void **)&t->entries, he.data(), he.size() * sizeof(TrEntry));
  if (e == cudaSuccess) e = up((void **)&t->pieces, hp.data(), hp.size() * sizeof(TrPiece));
  if (e == cudaSuccess) e = up((void **)&t->task_group, htask.data(), htask.size() * 4);
  if (e != cudaSuccess) {
    tkb_trace_table_destroy(t);
    return tkb_set_error(ctx, e == cudaErrorMemoryAllocation ? TKB_ERR_OOM : TKB_ERR_CUDA,
                         std::string("trace table upload: ") + cudaGetErrorString(e));
  }
  *out = t;
  return TKB_OK;
}

extern "C" int tkb_trace_table_destroy(tkb_trace_table *t) {
  if (!t) return TKB_OK;
  cudaFree(t->groups);
  cudaFree(t->entries);
  cudaFree(t->pieces);
  cudaFree(t->task_group);
  delete t;
  return TKB_OK;
}

namespace {
template <typename T, bool CONJ>
cudaError_t trace_launch(tkb_ctx *ctx, const tkb_trace_table *t, void *dst, const void *src, CDbl a, CDbl b, int bz) {
  const bool few = t->nfree <= 2, multi = t->ntrace > 1;
  auto k = few ? (multi ? trace_kernel<T, CONJ, 2, true> : trace_kernel<T, CONJ, 2, false>)
               : (multi ? trace_kernel<T, CONJ, TKB_MAX_IND, true> : trace_kernel<T, CONJ, TKB_MAX_IND, false>);
  const int grid = (int)std::min<int64_t>(t->ntasks, INT32_MAX);
  return launch_pdl(k, dim3(grid), dim3(kTrThreads), 0, ctx->stream, t->groups, t->entries, t->pieces, t->task_group,
                    t->ntasks, t->nfree, t->ntrace, (T *)dst, (const T *)src, a, b, bz);
}
}  // namespace

extern "C" int tkb_tracetransform(tkb_ctx *ctx, const tkb_trace_table *t, int dtype, void *dst,
                                  const void *src, tkb_scalar alpha, tkb_scalar beta, int conj) {
  if (!ctx || !t) return TKB_ERR_ARG;
  if (t->owner != ctx) return tkb_set_error(ctx, TKB_ERR_ARG, "trace table belongs to another context");
  if (t->ntasks == 0) return TKB_OK;
  if (!dst || !src) return tkb_set_error(ctx, TKB_ERR_ARG, "null data pointer");
  const CDbl a{alpha.re, alpha.im}, b{beta.re, beta.im};
  const int bz = (beta.re == 0.0 && beta.im == 0.0) ? 1 : 0;
  cudaError_t e = cudaSuccess;
  if (dtype == TKB_F64) {
    if (alpha.im != 0.0 || beta.im != 0.0)
      return tkb_set_error(ctx, TKB_ERR_ARG, "complex scalar with real data");
    e = trace_launch<double, false>(ctx, t, dst, src, a, b, bz);
  } else if (dtype == TKB_C128) {
    e = conj ? trace_launch<double2, true>(ctx, t, dst, src, a, b, bz)
             : trace_launch<double2, false>(ctx, t, dst, src, a, b, bz);
  } else {
    return tkb_set_error(ctx, TKB_ERR_ARG, "unknown dtype");
  }
  TKB_CUDA_TRY(ctx, e);
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}
