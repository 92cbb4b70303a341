// Weighted block reductions for norm / inner / tr (src/tensors/linalg.jl:257-282, 319-327;
// src/tensors/vectorinterface.jl:114-130): Σ_c dim(c)·f(block_c), accumulated in FP64.
//
// One launch: a warp takes a contiguous range of the segments' element space and walks the
// segments in it, the weight applied once per segment piece; the CTA that arrives last on a
// counter adds the partial sums in CTA order (deterministic: which CTA that is does not
// matter) and writes the result, to host memory where the caller waits for it. A segment is a round trip
// to its record and to its elements however short it is, so in the element space every segment is followed by
// kRedSegPad places without an element, which spread many short ones (the blocks of a tensor with many
// sectors, all diagonals of a trace) over warps and CTAs. The norm of 1001 blocks of one element takes 7 us (487
// when the whole CTA walked them one by one), the trace of 147 blocks of 40 x 40 7 us (49).
//
// The counter word holds the launch's ticket above the arrivals. A CTA first raises the word to its
// launch's ticket, so every launch counts from zero whatever an earlier one left there (launches overlap
// where the caller gives the context another stream in between), without a memset of 2.5 us in front.
// Launches take the counters and partial sums of a ring in turn, so those that overlap share neither.
//
// Bound: HBM. A thread keeps eight accesses in flight (four of x and four of y for INNER, where eight
// of each took 41 us), 16 bytes each where the piece is contiguous and aligned alike in both
// vectors. On 10.6 M doubles (cold caches, alone): inner 36 us (4.7 TB/s; 52 with one 8-byte access
// in flight and the weight applied per element), norm 22.5 us (3.8 TB/s; 45). The second launch that
// added the partial sums took another 4 us and the copy of the result a transfer of its own.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "tkb_internal.h"

namespace {

constexpr int RT = 256;
// accesses of each vector in flight per thread: eight in all
template <int KIND>
constexpr int kRedBatch = KIND == TKB_INNER ? 4 : 8;

struct Acc {
  double re, im;
};
template <int KIND>
__device__ __forceinline__ void term(Acc &a, double x, double y) {
  if constexpr (KIND == TKB_NORM2) a.re = fma(x, x, a.re);
  else if constexpr (KIND == TKB_INNER) a.re = fma(x, y, a.re);
  else a.re += x;
}
template <int KIND>
__device__ __forceinline__ void term(Acc &a, double2 x, double2 y) {
  if constexpr (KIND == TKB_NORM2) {
    a.re = fma(x.x, x.x, fma(x.y, x.y, a.re));
  } else if constexpr (KIND == TKB_INNER) {  // conj(x)·y
    a.re = fma(x.x, y.x, fma(x.y, y.y, a.re));
    a.im = fma(x.x, y.y, fma(-x.y, y.x, a.im));
  } else {
    a.re += x.x;
    a.im += x.y;
  }
}
// a pair of real elements read as one 16-byte value
template <int KIND>
__device__ __forceinline__ void term_pair(Acc &a, double2 x, double2 y) {
  term<KIND>(a, x.x, y.x);
  term<KIND>(a, x.y, y.y);
}

__device__ __forceinline__ double2 block_sum(double2 v) {
  __shared__ double2 red[RT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double2 r = make_double2(0.0, 0.0);
  if (threadIdx.x == 0)
    for (int w = 0; w < RT / 32; ++w) { r.x += red[w].x; r.y += red[w].y; }
  __syncthreads();
  return r;
}

// Σ over n values x[i·stride] (and y) of a warp, the thread's share, in independent sums
template <int KIND, typename T, typename F>
__device__ __forceinline__ void piece_sum(const T *__restrict__ x, const T *__restrict__ y, int64_t n, int64_t stride,
                                          Acc (&a)[kRedBatch<KIND>], F &&add) {
  for (int64_t i0 = threadIdx.x & 31; i0 < n; i0 += 32 * kRedBatch<KIND>) {
    T xv[kRedBatch<KIND>], yv[kRedBatch<KIND>];
#pragma unroll
    for (int q = 0; q < kRedBatch<KIND>; ++q) {
      const int64_t i = i0 + q * 32;
      if (i < n) {
        xv[q] = __ldg(x + i * stride);
        yv[q] = KIND == TKB_INNER ? __ldg(y + i * stride) : xv[q];
      }
    }
#pragma unroll
    for (int q = 0; q < kRedBatch<KIND>; ++q)
      if (i0 + q * 32 < n) add(a[q], xv[q], yv[q]);
  }
}

template <int KIND, typename T>
__global__ void __launch_bounds__(RT)
    reduce_kernel(const RSeg *__restrict__ segs, const int64_t *__restrict__ seg_begin, int64_t nseg, int64_t span,
                  const T *__restrict__ x, const T *__restrict__ y, double2 *__restrict__ partial,
                  unsigned long long *arrived, unsigned long long ticket, double *out) {
  __shared__ int last;
  pdl_wait();  // the vectors, the partial sums and the counter belong to earlier kernels too
  pdl_trigger();
  if (threadIdx.x == 0) atomicMax(arrived, ticket);
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = (int64_t)gridDim.x * (RT / 32);
  const int64_t per = (span + nwarps - 1) / nwarps;
  const int64_t wb = ((int64_t)blockIdx.x * (RT / 32) + threadIdx.x / 32) * per;
  const int64_t we = min(span, wb + per);
  double2 acc = make_double2(0.0, 0.0);
  if (wb < we) {
    // the last segment that begins at or before wb, in steps of 32 candidates
    int64_t s = 0;
    for (int64_t left = nseg; left > 1;) {
      const int64_t step = (left + 31) / 32, at = lane * step;
      const unsigned before = __ballot_sync(0xffffffffu, at < left && seg_begin[s + min(at, left - 1)] <= wb);
      const int64_t k = (31 - __clz(before)) * step;  // lane 0's candidate begins before wb
      s += k;
      left = min(step, left - k);
    }
    RSeg next = segs[s];
    int64_t next_begin = seg_begin[s];
    for (; s < nseg && next_begin < we; ++s) {
      const RSeg sg = next;
      const int64_t begin = next_begin;
      if (s + 1 < nseg) {  // the next record arrives while this segment is summed
        next = segs[s + 1];
        next_begin = seg_begin[s + 1];
      }
      const int64_t b = max(wb, begin), e = min(we, begin + sg.count);
      if (b >= e) continue;
      const int64_t at = sg.off + (b - begin) * sg.stride;
      const T *xp = x + at, *yp = KIND == TKB_INNER ? y + at : xp;
      int64_t n = e - b;
      Acc a[kRedBatch<KIND>];
#pragma unroll
      for (int q = 0; q < kRedBatch<KIND>; ++q) a[q] = Acc{0.0, 0.0};
      auto one = [](Acc &c, T u, T v) { term<KIND>(c, u, v); };
      bool pairs = false;
      if constexpr (sizeof(T) == 8) {
        pairs = sg.stride == 1 && n >= 2 && (((uintptr_t)xp ^ (uintptr_t)yp) & 15) == 0;
        if (pairs) {
          const int head = ((uintptr_t)xp & 15) ? 1 : 0;
          const int64_t np = (n - head) / 2;
          const int tail = (int)(n - head - 2 * np);
          if (lane == 0) {
            if (head) one(a[0], xp[0], yp[0]);
            if (tail) one(a[0], xp[n - 1], yp[n - 1]);
          }
          piece_sum<KIND, double2>(reinterpret_cast<const double2 *>(xp + head),
                                   reinterpret_cast<const double2 *>(yp + head), np, 1, a,
                                   [](Acc &c, double2 u, double2 v) { term_pair<KIND>(c, u, v); });
        }
      }
      if (!pairs) piece_sum<KIND, T>(xp, yp, n, sg.stride, a, one);
#pragma unroll
      for (int h = kRedBatch<KIND> / 2; h > 0; h >>= 1)  // pairwise
#pragma unroll
        for (int q = 0; q < h; ++q) {
          a[q].re += a[q + h].re;
          a[q].im += a[q + h].im;
        }
      acc.x = fma(sg.weight, a[0].re, acc.x);
      acc.y = fma(sg.weight, a[0].im, acc.y);
    }
  }
  const double2 r = block_sum(acc);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = r;
    __threadfence();
    last = atomicAdd(arrived, 1ull) == ticket + gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double2 sum = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < (int)gridDim.x; i += RT) {
    const double2 p = __ldcg(&partial[i]);
    sum.x += p.x;
    sum.y += p.y;
  }
  const double2 res = block_sum(sum);
  if (threadIdx.x == 0) {
    *arrived = 0;  // every CTA has arrived: free for the next launch (of a graph: with the same ticket)
    out[0] = res.x;
    out[1] = res.y;
  }
}

template <typename T>
cudaError_t reduce_launch(int kind, int nb, cudaStream_t st, const RSeg *segs, const int64_t *begin, int64_t nseg,
                          int64_t span, const void *x, const void *y, double2 *partial, unsigned long long *arrived,
                          unsigned long long ticket, double *out) {
  auto k = kind == TKB_NORM2 ? reduce_kernel<TKB_NORM2, T>
           : kind == TKB_INNER ? reduce_kernel<TKB_INNER, T>
                               : reduce_kernel<TKB_TRACE, T>;
  return launch_pdl(k, dim3(nb), dim3(RT), 0, st, segs, begin, nseg, span, (const T *)x, (const T *)y, partial,
                    arrived, ticket, out);
}

}  // namespace

// ---- allocation-free variant ------------------------------------------------------------
// Scratch for tkb_reduce_noalloc: segment table, prefix sums, per-CTA partials and the
// result, in one file-scope device array that every GPU loading the library holds until
// the process exits. Host code only sees a stand-in for this symbol; its device address
// comes from cudaGetSymbolAddress, taken once per device.
namespace {
constexpr int64_t kNoAllocMaxSeg = 1024;
constexpr int kNoAllocMaxCta = 1024;
constexpr size_t kNoAllocSegBytes = kNoAllocMaxSeg * sizeof(RSeg);                 // 32 KiB
constexpr size_t kNoAllocBeginOff = kNoAllocSegBytes;
constexpr size_t kNoAllocPartialOff = (kNoAllocBeginOff + (kNoAllocMaxSeg + 1) * 8 + 255) / 256 * 256;
constexpr size_t kNoAllocResultOff = kNoAllocPartialOff + kNoAllocMaxCta * sizeof(double2);
constexpr size_t kNoAllocCountOff = kNoAllocResultOff + 128;  // arrival counter
constexpr size_t kNoAllocBytes = kNoAllocResultOff + 256;                          // ~57 KiB
}  // namespace

static __device__ __align__(256) unsigned char tkb_noalloc_scratch[kNoAllocBytes];

namespace {
std::mutex g_noalloc_mu;
void *g_noalloc_ptr[64] = {nullptr};
}  // namespace

extern "C" int tkb_reduce_noalloc(int device, void *stream, int kind, int dtype, const void *x,
                                  const void *y, int64_t len, int64_t nseg, const int64_t *off,
                                  const int64_t *count, const int64_t *stride, const double *weight,
                                  double *host_out) {
  if (kind < TKB_NORM2 || kind > TKB_TRACE) return tkb_set_error(nullptr, TKB_ERR_ARG, "unknown reduction");
  if (dtype != TKB_F64 && dtype != TKB_C128) return tkb_set_error(nullptr, TKB_ERR_ARG, "unknown dtype");
  if (!host_out) return tkb_set_error(nullptr, TKB_ERR_ARG, "null output");
  if (device < 0 || device >= 64) return tkb_set_error(nullptr, TKB_ERR_ARG, "device out of range");
  if (nseg < 0 || nseg > kNoAllocMaxSeg)
    return tkb_set_error(nullptr, TKB_ERR_SIZE,
                         "tkb_reduce_noalloc supports at most 1024 segments (got " +
                             std::to_string(nseg) + "); use tkb_reduce for larger tensors");
  if (nseg > 0 && (!off || !count || !stride || !weight))
    return tkb_set_error(nullptr, TKB_ERR_ARG, "null segment array");
  // validation (overflow-safe: count − 1 is compared with the room left after off)
  int64_t total = 0;
  for (int64_t s = 0; s < nseg; ++s) {
    if (count[s] < 0 || off[s] < 0 || stride[s] < 0)
      return tkb_set_error(nullptr, TKB_ERR_ARG, "invalid segment");
    if (count[s] > 0 && !tkb_segment_in_bounds(off[s], count[s], stride[s], len))
      return tkb_set_error(nullptr, TKB_ERR_SIZE, "segment outside the data vector");
    total += count[s];
  }
  if (total > 0 && (!x || (kind == TKB_INNER && !y)))
    return tkb_set_error(nullptr, TKB_ERR_ARG, "null data");

  int prev = 0;
  if (cudaGetDevice(&prev) != cudaSuccess) prev = device;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return tkb_set_error(nullptr, TKB_ERR_CUDA, cudaGetErrorString(e));
  unsigned char *base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[device]) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, tkb_noalloc_scratch);
      if (e != cudaSuccess) {
        cudaSetDevice(prev);
        return tkb_set_error(nullptr, TKB_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      }
      g_noalloc_ptr[device] = p;
    }
    base = static_cast<unsigned char *>(g_noalloc_ptr[device]);
  }
  cudaStream_t st = (cudaStream_t)stream;
  RSeg *dsegs = reinterpret_cast<RSeg *>(base);
  int64_t *dbegin = reinterpret_cast<int64_t *>(base + kNoAllocBeginOff);
  double2 *dpart = reinterpret_cast<double2 *>(base + kNoAllocPartialOff);
  double *dres = reinterpret_cast<double *>(base + kNoAllocResultOff);
  e = cudaSuccess;
  if (total == 0) {
    host_out[0] = 0.0;
    host_out[1] = 0.0;
  } else {
    // The segment table and its prefix sums go up in chunks staged in small stack buffers
    // (a few KiB: callers such as finalizers may run on small stacks). The sources are pageable
    // host memory, so each copy has read its buffer when cudaMemcpyAsync returns and the buffer
    // can be refilled.
    constexpr int64_t kChunk = 64;
    RSeg segs[kChunk];
    int64_t begin[kChunk + 1];
    int64_t run = 0;
    for (int64_t s0 = 0; s0 < nseg && e == cudaSuccess; s0 += kChunk) {
      const int64_t n = std::min<int64_t>(kChunk, nseg - s0);
      for (int64_t q = 0; q < n; ++q) {
        const int64_t s = s0 + q;
        segs[q] = {off[s], count[s], stride[s], weight[s]};
        begin[q] = run;
        run += count[s] + kRedSegPad;
      }
      begin[n] = run;
      e = cudaMemcpyAsync(dsegs + s0, segs, n * sizeof(RSeg), cudaMemcpyHostToDevice, st);
      // the prefix sums overlap by one entry between chunks (the same value is written twice)
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(dbegin + s0, begin, (n + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st);
    }
    const int nb = (int)std::min<int64_t>((run + 4095) / 4096, kNoAllocMaxCta);
    if (e == cudaSuccess) {
      // calls that overlap share the counter: each starts it anew, so that none spoils those after it
      auto *arrived = reinterpret_cast<unsigned long long *>(base + kNoAllocCountOff);
      const unsigned long long ticket = kRedTicket;
      e = cudaMemsetAsync(arrived, 0, sizeof(*arrived), st);
      if (e == cudaSuccess)
        e = dtype == TKB_F64
                ? reduce_launch<double>(kind, nb, st, dsegs, dbegin, nseg, run, x, y, dpart, arrived, ticket, dres)
                : reduce_launch<double2>(kind, nb, st, dsegs, dbegin, nseg, run, x, y, dpart, arrived, ticket, dres);
    }
    if (e == cudaSuccess) {
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(host_out, dres, 2 * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  cudaSetDevice(prev);
  if (e != cudaSuccess) return tkb_set_error(nullptr, TKB_ERR_CUDA, cudaGetErrorString(e));
  return TKB_OK;
}

int tkb_reduce_launch(tkb_ctx *ctx, const tkb_rplan *p, int kind, int dtype, const void *x,
                      const void *y, double *dev_out) {
  const int nb = p->nblocks_launch;  // at most kRedCtasPerSm per SM
  if (p->total == 0) {
    TKB_CUDA_TRY(ctx, cudaMemsetAsync(dev_out, 0, 2 * sizeof(double), ctx->stream));
    return TKB_OK;
  }
  const uint64_t call = ctx->red_calls.fetch_add(1);
  const int slot = (int)(call % kRedSlots);
  const unsigned long long ticket = (call + 1) * kRedTicket;
  auto *arrived = reinterpret_cast<unsigned long long *>(ctx->red_scratch) + slot;
  double2 *partial = reinterpret_cast<double2 *>(ctx->red_scratch + kRedSlots * sizeof(*arrived)) +
                     (size_t)slot * ctx->num_sms * kRedCtasPerSm;
  // a captured launch runs with its ticket of today whatever tickets came between: it starts from zero
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  TKB_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
  if (cap != cudaStreamCaptureStatusNone)
    TKB_CUDA_TRY(ctx, cudaMemsetAsync(arrived, 0, sizeof(*arrived), ctx->stream));
  TKB_CUDA_TRY(ctx, dtype == TKB_F64
                        ? reduce_launch<double>(kind, nb, ctx->stream, p->segs, p->seg_begin, p->nseg, p->span, x, y,
                                                partial, arrived, ticket, dev_out)
                        : reduce_launch<double2>(kind, nb, ctx->stream, p->segs, p->seg_begin, p->nseg, p->span, x, y,
                                                 partial, arrived, ticket, dev_out));
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}
