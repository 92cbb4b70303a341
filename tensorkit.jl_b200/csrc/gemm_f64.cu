// Plain FP64 / ComplexF64 grouped block GEMM: one launch for all coupled-sector blocks of a
// TensorKit mul! (src/tensors/linalg.jl:330-370).
//
// Tensor path: FP64 DMMA (mma.sync m16n8k8; four of them per complex fragment pair). tcgen05 has no
// f64 kind, so the double-precision tensor pipe is reached through DMMA; the split-precision
// path (gemm_split.cu) is the tcgen05 one.
//
// Work decomposition (tkb_gemm_plain_prepare): 64×64 output tiles (64×32 complex; 32×32 where those would leave
// part of the chip idle), whose K loops are cut into pieces (split K) where that evens out the CTAs'
// shares. Every CTA has a fixed list of tasks (tile, K range). A piece of a split tile stores its
// FP64 partial tile; the piece that arrives last on the tile's counter adds all partials in piece
// order (deterministic, no piece waits for another) and applies α, β.
//
// CTA: 4 warps in a 2×2 grid, m16n8k8 tiles, BK = 16, a three-stage cp.async ring (two stages in
// flight while one is consumed; one barrier per K step; a stage's DMMA are issued before the refill
// copies). The ring runs through all tasks of the CTA without a break: the next tile's first stages
// arrive while the last one's values are stored. Operand tiles are copied in 16-byte pairs when the
// block's layout keeps pairs aligned (op N, even offsets and leading dimensions, 16-byte aligned base),
// else in 8-byte elements; elements outside the block are zero-filled, so any lda/offset parity
// works. Complex blocks copy whole 16-byte elements and issue four real DMMA per fragment pair.
//
// What bounds it: the DMMA pipe runs m16n8k8 at 64 cycles per SM sub-partition (37 TFLOP/s measured on
// B200), and every instruction issued beside it costs: with addresses and bounds resolved once per
// task one 4096³ block runs at 33.7 TFLOP/s (30.1 when each copy worked out its own address), one
// 4095³ block (8-byte copies) at 32.8 (26.8), one complex 2048³ block at 32.7 (30.4). The epilogue
// keeps one pointer per column of a thread: 9 blocks of K ≤ 256 and a 59 MB output take 152 us (176 with an
// address per element, 37 us of it in the epilogues). Taken back: fragments of the next sub-step loaded ahead of the DMMA (517 instead of
// 489 us on a U(1) effective Hamiltonian; the DMMA wait for the loads issued before them).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "tkb_internal.h"

namespace {

constexpr int BK = 16;  // K positions per stage

struct CDbl {
  double x, y;
};

// one task of the plain kernels: an output tile and a range of its K steps
struct PTask {
  int32_t block, m0, n0, kind;  // kind 0: products, 1: β-scale only (k = 0)
  int32_t kb, ke;               // K steps [kb, ke) of BK
  int32_t slot, nsplit;         // split K: counter slot, pieces of the tile (1 = unsplit)
  int32_t sid, pbase;           // piece index, first partial buffer of the tile
};

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
// 16-byte copy of which the first `bytes` (0, 8 or 16) come from global memory, the rest zero
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, int bytes) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Timeline build (-DTKB_TIMELINE): per CTA of the real kernel, global-timer stamps (ns) at entry
// (0), after the grid-dependency wait (1), after the first task's K loop (2) and split-K
// arrival (3), at exit (4); slot 5 counts the CTA's tasks, slot 6 holds the first task's
// pieces and whether it was the last to arrive (2·nsplit + last). Read with
// tkb_timeline_read_plain; the default build compiles every stamp away.
#ifdef TKB_TIMELINE
constexpr int kPlTlCtas = 512, kPlTlSlots = 8;
__device__ unsigned long long tkb_tl_plain[kPlTlCtas * kPlTlSlots];
__device__ __forceinline__ unsigned long long pl_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
#define PL_SET(k, v)                                                                         \
  do {                                                                                       \
    if (threadIdx.x == 0 && blockIdx.x < kPlTlCtas) tkb_tl_plain[blockIdx.x * kPlTlSlots + (k)] = (v); \
  } while (0)
#else
#define PL_SET(k, v) ((void)0)
#endif
#define PL_STAMP(k) PL_SET(k, pl_now())

// D(16×8) += A(16×8) B(8×8), FP64. Lane (g = lane/4, t = lane%4): a = A[g][t], A[g+8][t],
// A[g][t+4], A[g+8][t+4]; b = B[t][g], B[t+4][g]; c = D[g][2t], D[g][2t+1], D[g+8][2t],
// D[g+8][2t+1] (checked against a host product on the device)
__device__ __forceinline__ void dmma16(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
// D = A B
__device__ __forceinline__ void dmma16_first(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=d"(c[0]), "=d"(c[1]), "=d"(c[2]), "=d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]), "d"(0.0));
}

// ---- tiled kernel ------------------------------------------------------------------------
// Where the products of one output value meet. One accumulator that takes every product of a long K loses more
// in rounding than several that are added in the end (64x64 sampled values of ten products of K = 31 - 1736
// against long double: up to 1.9 times the error of Halves real, 1.7 complex).
//   One:    a single accumulator (64×32 complex tiles, which have no registers left)
//   Halves: one for each half of a stage
//   Stage:  a stage is summed from zero, then added. An FP64 addition per value and stage takes 6 % of the pipe
//           that the DMMA need, which does not show while the launch waits for latency (32×32 real tiles)
//   Stages: the same every fourth stage (32×32 complex tiles, which also run launches bound by the DMMA: 69.7 us
//           for an SU(2) environment update at V dim 2406, 69.6 with One, 82.4 with Stage)
enum class Sum { One, Halves, Stage, Stages };
constexpr int kSumStages = 4;

// Tile shape of a kernel for elements E (double, or double2 for complex data): BMxBN output tile, warps
// of WMxWN (m16n8k8 fragments). The pitches spread the fragments of a warp over the banks.
template <typename E_, int BM_, int BN_, int WM_, int WN_, int NST_, int MINB_, Sum SUM_>
struct TileCfg {
  using E = E_;
  static constexpr bool CPLX = sizeof(E) == 16;
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, NST = NST_, MINB = MINB_;
  static constexpr int WARPS_M = BM / WM, WARPS = (BM / WM) * (BN / WN), THREADS = 32 * WARPS;
  static constexpr int MI = WM / 16, NI = WN / 8, NV = MI * NI * (CPLX ? 8 : 4);  // NV: accumulators per thread
  static constexpr Sum SUM = SUM_;
  static constexpr bool BETA_KERNEL = SUM != Sum::One;  // kernels of their own without and with β
  static constexpr int NACC = SUM == Sum::Halves || SUM == Sum::Stages ? 2 * NV : NV;  // with the second set
  // pitches of an operand's tile in a stage: [k][outer] or [outer][k] (see TileCopy)
  static constexpr int PA = BM + (CPLX ? 2 : 4), PB = BN + (CPLX ? 2 : 4), PK = BK + 4;
  // (op(A): [k][row] real, either complex; op(B): [col][k] real, either complex)
  static constexpr int A_ELEMS = CPLX && BM * PK > BK * PA ? BM * PK : BK * PA;
  static constexpr int B_ELEMS = CPLX && BK * PB > BN * PK ? BK * PB : BN * PK, STAGE = A_ELEMS + B_ELEMS;
  static constexpr size_t SMEM = (size_t)NST * STAGE * sizeof(E);
};

// Copies of one operand's tiles, resolved once per task: the thread's first source element, the
// step to its next copies of a stage and to the next stage. Copies of rows (columns) outside the block read
// nothing and fill zeros; so do K positions beyond the block. Tiles inside the block on both counts
// take a path without the tests: one address step and one copy per element (or pair), the place
// in the stage an immediate offset. Instruction issue, not the copies' latency, is what a stage
// costs besides its DMMA.
//   kind 0: the tile's outer index (rows of op(A), columns of op(B)) is contiguous in memory
//   kind 1: K is contiguous
//   kind 2: 16-byte pairs along the contiguous direction that the stage keeps contiguous too
// In the stage, real tiles are always [k][outer] (op(A), pitch PO) or [outer][k] (op(B), pitch PK). Complex tiles keep
// the direction that is contiguous in memory contiguous: 16-byte pieces that scatter in the stage are fetched one by
// one (an adjoint op(A) with the fixed layout: twice the L2 requests, 296 instead of 249 us for 1500 x 400 x 1500;
// 8-byte pieces do not suffer, and a second layout made small real products 0.8 us slower).
template <typename E, int T, int OUTER, bool IS_A, int PO, int PK>
struct TileCopy {
  const E *p, *base;  // base: the operand's first element (where copies that read nothing point)
  int64_t dr, dk;    // elements: between the copies of a stage, between stages
  int kind, o, ext;  // outer position of the first copy in the block, the block's extent (clamped)
  int l0, s0;        // K position and stage offset of the first copy
  bool inside;       // the whole tile lies inside the block

  // thread layout of a kind: first (outer, K) position and the steps between its copies
  template <int KIND>
  struct Lay {
    static constexpr int COPIES = KIND == 2 ? OUTER * BK / (2 * T) : OUTER * BK / T;
    static constexpr bool ALONG_K = KIND == 2 ? !IS_A : KIND == 1;  // neighbouring threads step along K
    static constexpr int W = KIND == 2 ? 2 : 1;
    static constexpr int LINE = (ALONG_K ? BK : OUTER) / W;         // threads per contiguous run
    static constexpr int DO = ALONG_K ? T / LINE : 0, DL = ALONG_K ? 0 : T / LINE;
    static constexpr bool K_IN = sizeof(E) == 16 ? KIND == 1 : !IS_A;  // the stage is [outer][k]
    static constexpr int DS = K_IN ? DO * PK + DL : DL * PO + DO;
    static_assert(T % LINE == 0, "whole runs per pass");
  };
  template <int KIND>
  __device__ __forceinline__ void init_kind(int64_t so, int64_t sk, int64_t o0, int64_t kbeg) {
    using L = Lay<KIND>;
    const int a = (threadIdx.x % L::LINE) * L::W, b = threadIdx.x / L::LINE;
    const int oo = L::ALONG_K ? b : a;
    l0 = L::ALONG_K ? a : b;
    p = base + (o0 + oo) * so + (kbeg + l0) * sk;
    dr = L::DO * so + L::DL * sk;
    s0 = L::K_IN ? oo * PK + l0 : l0 * PO + oo;
    o = oo;
  }
  __device__ __forceinline__ void init(const E *X, int64_t off, int64_t ld, bool outer_contig, int64_t o0,
                                       int64_t extent, int64_t kbeg, bool pairs) {
    const int64_t so = outer_contig ? 1 : ld, sk = outer_contig ? ld : 1;
    base = X + off;
    dk = BK * sk;
    const int64_t rest = extent - o0;  // outer positions from the tile's first on
    inside = rest >= OUTER;
    ext = inside ? OUTER : (int)rest;
    kind = pairs && outer_contig == IS_A ? 2 : outer_contig ? 0 : 1;
    if (kind == 0) init_kind<0>(so, sk, o0, kbeg);
    else if (kind == 1) init_kind<1>(so, sk, o0, kbeg);
    else if constexpr (sizeof(E) == 8) init_kind<2>(so, sk, o0, kbeg);
  }
  static __device__ __forceinline__ void copy(E *d, const E *q, bool v) {
    if constexpr (sizeof(E) == 8) cp_async8(d, q, v);
    else cp_async16(d, q, v ? 16 : 0);
  }
  template <int KIND>
  __device__ __forceinline__ void issue_kind(E *stage, int64_t left) {
    using L = Lay<KIND>;
    E *d = stage + s0;
    const E *q = p;
    if (inside && left >= BK) {
#pragma unroll
      for (int r = 0; r < L::COPIES; ++r, q += dr) {
        if constexpr (KIND == 2) cp_async16(d + r * L::DS, q, 16);
        else copy(d + r * L::DS, q, true);
      }
    } else {
#pragma unroll
      for (int r = 0; r < L::COPIES; ++r, q += dr) {
        const int oo = o + r * L::DO, l = l0 + r * L::DL;
        if constexpr (KIND == 2) {  // the pair's second element may lie outside
          const bool v = oo < ext && l < left;
          const bool w = L::ALONG_K ? l + 1 < left : oo + 1 < ext;
          cp_async16(d + r * L::DS, v ? q : base, v ? (w ? 16 : 8) : 0);
        } else {
          const bool v = oo < ext && l < left;
          copy(d + r * L::DS, v ? q : base, v);
        }
      }
    }
  }
  // the copies of the next stage into `stage`; left: K positions of the block from this stage on
  __device__ __forceinline__ void issue(E *stage, int64_t left) {
    if (kind == 0) issue_kind<0>(stage, left);
    else if (kind == 1) issue_kind<1>(stage, left);
    else if constexpr (sizeof(E) == 8) issue_kind<2>(stage, left);
    p += dk;
  }
};

// 16-byte pairs are usable for an operand in op N whose offset and leading dimension are even
// (the base pointer's alignment is checked at launch)
__device__ __forceinline__ int vec_flags(const GBlock &b, int base_ok) {
  int v = 0;
  if ((base_ok & 1) && b.opA == TKB_OP_N && !(b.offA & 1) && !(b.lda & 1)) v |= 1;
  if ((base_ok & 2) && b.opB == TKB_OP_N && !(b.offB & 1) && !(b.ldb & 1)) v |= 2;
  return v;
}

// Split-K: store this piece's values (q-major: value q of every thread, so warps store
// contiguous runs), count the arrival; the last piece of the tile reads all partials in piece
// order and returns true with their sum in v. Unsplit tiles return true with v unchanged.
template <int NV, int NT>
__device__ __forceinline__ bool splitk_reduce(const PTask &t, double (&v)[NV], double *part, int *pcnt,
                                              int *ticket) {
  if (t.nsplit <= 1) return true;
  const int tid = threadIdx.x;
  double *mine = part + (int64_t)(t.pbase + t.sid) * (NV * NT);
#pragma unroll
  for (int q = 0; q < NV; ++q) __stcg(&mine[q * NT + tid], v[q]);
  __threadfence();
  __syncthreads();
  if (tid == 0) *ticket = atomicAdd(&pcnt[t.slot], 1);
  __syncthreads();
  const bool last = *ticket == t.nsplit - 1;
  __syncthreads();  // ticket is rewritten by the next task
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < NV; ++q) v[q] = 0.0;
  for (int sp = 0; sp < t.nsplit; ++sp) {  // piece order: deterministic sum
    const double *src = part + (int64_t)(t.pbase + sp) * (NV * NT);
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] += __ldcg(&src[q * NT + tid]);
  }
  if (tid == 0) pcnt[t.slot] = 0;  // every piece has arrived: the counter is free for the next launch
  return true;
}

// v with its sign flipped where mask is 0x80000000
__device__ __forceinline__ double flip(double v, int mask) {
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

// The products of one stage: op(A) tile sa and op(B) tile sb from the thread's row i and column j on. AK, BKC: the tile
// is [outer][k]; both layouts spread the values that a warp reads at once over all banks.
template <typename CFG, bool AK, bool BKC>
__device__ __forceinline__ void stage_products(double (&acc)[CFG::NACC], const typename CFG::E *sa,
                                               const typename CFG::E *sb, int i, int j, int t, int conjA, int conjB) {
  constexpr int AR = AK ? CFG::PK : 1, AL = AK ? 1 : CFG::PA, BC = BKC ? CFG::PK : 1, BL = BKC ? 1 : CFG::PB;
  sa += i * AR + t * AL;
  sb += j * BC + t * BL;
  constexpr bool STAGE = CFG::SUM == Sum::Stage;
  [[maybe_unused]] double fresh[STAGE ? CFG::NV : 1];
#pragma unroll
  for (int kk = 0; kk < BK; kk += 8) {
    const bool first = STAGE && kk == 0;
    double *sum = STAGE ? fresh : CFG::SUM == Sum::Halves && kk > 0 ? acc + CFG::NV : acc;
    auto product = [&](int v, const double (&a)[4], const double (&b)[2], bool from_zero) {
      double(&c)[4] = *reinterpret_cast<double(*)[4]>(sum + v);
      if (from_zero) dmma16_first(c, a, b);
      else dmma16(c, a, b);
    };
    if constexpr (!CFG::CPLX) {
      double af[CFG::MI][4], bf[CFG::NI][2];
#pragma unroll
      for (int mi = 0; mi < CFG::MI; ++mi)
#pragma unroll
        for (int q = 0; q < 4; ++q) af[mi][q] = sa[(kk + 4 * (q >> 1)) * AL + (mi * 16 + 8 * (q & 1)) * AR];
#pragma unroll
      for (int ni = 0; ni < CFG::NI; ++ni)
#pragma unroll
        for (int q = 0; q < 2; ++q) bf[ni][q] = sb[ni * 8 * BC + (kk + 4 * q) * BL];
#pragma unroll
      for (int mi = 0; mi < CFG::MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < CFG::NI; ++ni) product((mi * CFG::NI + ni) * 4, af[mi], bf[ni], first);
    } else {
      double br[CFG::NI][2], bi[CFG::NI][2];
#pragma unroll
      for (int ni = 0; ni < CFG::NI; ++ni)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const double2 v = sb[ni * 8 * BC + (kk + 4 * q) * BL];
          br[ni][q] = v.x;
          bi[ni][q] = flip(v.y, conjB);
        }
#pragma unroll
      for (int mi = 0; mi < CFG::MI; ++mi) {
        double ar[4], ai[4], an[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double2 v = sa[(kk + 4 * (q >> 1)) * AL + (mi * 16 + 8 * (q & 1)) * AR];
          ar[q] = v.x;
          ai[q] = flip(v.y, conjA);
          an[q] = flip(ai[q], (int)0x80000000);
        }
        // real products of all column fragments, then the imaginary ones: no two neighbours share
        // an accumulator
#pragma unroll
        for (int ni = 0; ni < CFG::NI; ++ni) {
          const int v = (mi * CFG::NI + ni) * 8;
          product(v, ar, br[ni], first);
          product(v + 4, ar, bi[ni], first);
        }
#pragma unroll
        for (int ni = 0; ni < CFG::NI; ++ni) {
          const int v = (mi * CFG::NI + ni) * 8;
          product(v, an, bi[ni], false);
          product(v + 4, ai, br[ni], false);
        }
      }
    }
  }
  if constexpr (STAGE) {
#pragma unroll
    for (int q = 0; q < CFG::NV; ++q) acc[q] += fresh[q];
  }
}

// BZ: β = 0 and the output is not read, in a kernel of its own (products of the sweeps 2 % faster, SU(2) update 51.2 ->
// 50.6 us). LargeTileC runs one kernel for both: alone, its β = 0 code came out at 194 registers instead of 226
// and one 2048³ block at 30.8 instead of 32.7 TFLOP/s.
template <typename CFG, bool BZ>
__global__ void __launch_bounds__(CFG::THREADS, CFG::MINB)
    gemm_plain_kernel(const GBlock *__restrict__ blocks, const PTask *__restrict__ tasks,
                      const int32_t *__restrict__ start, typename CFG::E *__restrict__ C,
                      const typename CFG::E *__restrict__ A, const typename CFG::E *__restrict__ B, CDbl alpha,
                      CDbl beta, double *__restrict__ part, int *__restrict__ pcnt, int base_ok) {
  using E = typename CFG::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  E *sm = reinterpret_cast<E *>(smem_raw);
  __shared__ int ticket;
  PL_STAMP(0);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp % CFG::WARPS_M) * CFG::WM, wn = (warp / CFG::WARPS_M) * CFG::WN;
  const int g = lane >> 2, t = lane & 3;
  const int t_begin = start[blockIdx.x], t_end = start[blockIdx.x + 1];
  // The stages of all the CTA's tasks form one stream through the ring: the copies run NST − 1 stages
  // ahead of the products and go on into the next task while this one finishes.
  TileCopy<E, CFG::THREADS, CFG::BM, true, CFG::PA, CFG::PK> ca;
  TileCopy<E, CFG::THREADS, CFG::BN, false, CFG::PB, CFG::PK> cb;
  int next = t_begin, ahead = 0;  // the next task to copy, stages of the current one not yet copied
  int64_t left = 0;               // K positions of its block from the next stage on
  auto advance = [&]() {
    while (ahead == 0 && next < t_end) {
      const PTask q = tasks[next++];
      ahead = q.kind == 0 ? q.ke - q.kb : 0;
      if (ahead == 0) continue;
      const GBlock &b = blocks[q.block];
      const int vec = CFG::CPLX ? 0 : vec_flags(b, base_ok);
      const int64_t k0 = (int64_t)q.kb * BK;
      ca.init(A, b.offA, b.lda, b.opA == TKB_OP_N, q.m0, b.m, k0, vec & 1);
      cb.init(B, b.offB, b.ldb, b.opB != TKB_OP_N, q.n0, b.n, k0, vec & 2);
      left = b.k - k0;
    }
  };
  auto produce = [&](int slot) {
    advance();
    if (ahead > 0) {
      ca.issue(sm + slot * CFG::STAGE, left);
      cb.issue(sm + slot * CFG::STAGE + CFG::A_ELEMS, left);
      left -= BK;
      --ahead;
    }
    cp_async_commit();  // one group per stage, possibly empty
  };
  advance();   // the task tables are static
  pdl_wait();  // operands, output and the split-K counters belong to earlier kernels too
  PL_STAMP(1);
#pragma unroll
  for (int st = 0; st < CFG::NST - 1; ++st) produce(st);
  int slot = 0;
  [[maybe_unused]] int ntask = 0;
  for (int ti = t_begin; ti < t_end; ++ti, ++ntask) {
    const PTask task = tasks[ti];
    // conjugation of an operand flips the sign of its imaginary part
    int conjA = 0, conjB = 0;
    if constexpr (CFG::CPLX) {
      conjA = blocks[task.block].opA == TKB_OP_C ? (int)0x80000000 : 0;
      conjB = blocks[task.block].opB == TKB_OP_C ? (int)0x80000000 : 0;
    }
    double acc[CFG::NACC];
#pragma unroll
    for (int q = 0; q < CFG::NACC; ++q) acc[q] = 0.0;
    const int nk = task.kind == 0 ? task.ke - task.kb : 0;
    auto k_loop = [&](auto ak, auto bk) {  // one loop per pair of layouts: no test inside
      auto stage = [&]() {
        cp_async_wait<CFG::NST - 2>();
        __syncthreads();  // this stage is visible to all; every warp is done with the slot before it
        const E *st = sm + slot * CFG::STAGE;
        stage_products<CFG, decltype(ak)::value, decltype(bk)::value>(acc, st, st + CFG::A_ELEMS, wm + g, wn + g, t,
                                                                      conjA, conjB);
        // the refill of the slot read in the previous iteration is issued while the DMMA execute
        produce(slot == 0 ? CFG::NST - 1 : slot - 1);
        slot = slot + 1 == CFG::NST ? 0 : slot + 1;
      };
      if constexpr (CFG::SUM == Sum::Stages) {  // loops in a loop: the stages stay free of the test
        for (int kt = 0; kt < nk;) {
          const int stop = min(nk, kt + kSumStages);
#pragma unroll 1
          for (; kt < stop; ++kt) stage();
#pragma unroll
          for (int q = 0; q < CFG::NV; ++q) {
            acc[CFG::NV + q] += acc[q];
            acc[q] = 0.0;
          }
        }
      } else {
        for (int kt = 0; kt < nk; ++kt) stage();
      }
    };
    constexpr std::true_type yes{};
    constexpr std::false_type no{};
    if constexpr (!CFG::CPLX) {
      k_loop(no, yes);
    } else {
      const bool ak = blocks[task.block].opA != TKB_OP_N, bk = blocks[task.block].opB == TKB_OP_N;
      if (bk) {
        if (!ak) k_loop(no, yes);
        else k_loop(yes, yes);
      } else {
        if (!ak) k_loop(no, no);
        else k_loop(yes, no);
      }
    }
    if constexpr (CFG::NACC > CFG::NV) {
#pragma unroll
      for (int q = 0; q < CFG::NV; ++q) acc[q] += acc[CFG::NV + q];
    }
    if (ntask == 0) PL_STAMP(2);
    if (ti + 1 == t_end) pdl_trigger();
    const bool fin = splitk_reduce<CFG::NV, CFG::THREADS>(task, *reinterpret_cast<double(*)[CFG::NV]>(acc), part, pcnt, &ticket);
    if (ntask == 0) {
      PL_STAMP(3);
      PL_SET(6, 2ull * task.nsplit + (fin ? 1 : 0));
    }
    if (!fin) continue;
    const GBlock &b = blocks[task.block];
    // epilogue: C = α·acc + β·C, column by column of the thread (column fragment q/2, column 2t + q%2);
    // its rows are 8 apart, so one pointer per column serves them all. Row h of column q is value
    // (h%2)·2 + q%2 of fragment (h/2, q/2) (complex: the imaginary part four values further)
    const int64_t i0 = task.m0 + wm + g, j0 = task.n0 + wn + 2 * t;
    const int rows = (int)min((int64_t)CFG::WM, b.m - i0);  // valid rows from i0 on (may be ≤ 0)
    const int cols = (int)min((int64_t)CFG::WN, b.n - j0);
    const int64_t ldc = b.ldc;
    E *pc = C + b.offC + i0 + j0 * ldc;
    auto value = [&](int q, int h) {  // α·(row h of column q)
      const double *f = &acc[((h >> 1) * CFG::NI + (q >> 1)) * (CFG::CPLX ? 8 : 4) + (h & 1) * 2 + (q & 1)];
      if constexpr (!CFG::CPLX) return alpha.x * f[0];
      else return make_double2(alpha.x * f[0] - alpha.y * f[4], alpha.x * f[4] + alpha.y * f[0]);
    };
    auto column = [](int q) { return (q / 2) * 8 + (q % 2); };
    if (BZ || (!CFG::BETA_KERNEL && beta.x == 0.0 && beta.y == 0.0)) {
#pragma unroll
      for (int q = 0; q < 2 * CFG::NI; ++q) {
        if (column(q) >= cols) continue;
        E *p = pc + column(q) * ldc;
#pragma unroll
        for (int h = 0; h < 2 * CFG::MI; ++h)
          if (h * 8 < rows) p[h * 8] = value(q, h);
      }
    } else if constexpr (!BZ) {
      // the old values of G columns are read at a time: 16 loads in flight (one column at a time, each column waited
      // for its own: 2048x64x2048 41.4 us with β, 36.3 so, 30.9 without)
      constexpr int G = CFG::CPLX || CFG::NI < 2 ? 2 : 4;
#pragma unroll
      for (int q0 = 0; q0 < 2 * CFG::NI; q0 += G) {
        E old[G][2 * CFG::MI];
#pragma unroll
        for (int q = q0; q < q0 + G; ++q)
#pragma unroll
          for (int h = 0; h < 2 * CFG::MI; ++h)
            if (column(q) < cols && h * 8 < rows) old[q - q0][h] = pc[column(q) * ldc + h * 8];
#pragma unroll
        for (int q = q0; q < q0 + G; ++q) {
          if (column(q) >= cols) continue;
          E *p = pc + column(q) * ldc;
#pragma unroll
          for (int h = 0; h < 2 * CFG::MI; ++h) {
            if (h * 8 < rows) {
              E r = value(q, h);
              const E &o = old[q - q0][h];
              if constexpr (!CFG::CPLX) {
                r = fma(beta.x, o, r);
              } else {
                r.x = fma(beta.x, o.x, fma(-beta.y, o.y, r.x));
                r.y = fma(beta.x, o.y, fma(beta.y, o.x, r.y));
              }
              p[h * 8] = r;
            }
          }
        }
      }
    }
  }
  cp_async_wait<0>();
  PL_SET(5, ntask);
  PL_STAMP(4);
}

// LargeTile: two CTAs of four 32×32 warps per SM (218 registers, 240 with β, with both accumulators; with one, three CTAs
// at 168 registers ran 4096³ at 32.5 instead of 33.8 TFLOP/s, eight 32×16 warps at 29.7). SmallTile: six CTAs of four 16×16 warps
// per SM, for launches whose 64×64 tiles would leave most of the chip to one CTA per SM, which spends
// 0.87 us per K step where its DMMA take 0.52.
using LargeTile = TileCfg<double, 64, 64, 32, 32, 3, 2, Sum::Halves>;
using SmallTile = TileCfg<double, 32, 32, 16, 16, 3, 6, Sum::Stage>;
// Complex fragments hold twice the values, so the large tile is half as wide (212 registers; 64×64 spills
// at the 128 registers of two CTAs).
using LargeTileC = TileCfg<double2, 64, 32, 32, 16, 3, 2, Sum::One>;
using SmallTileC = TileCfg<double2, 32, 32, 16, 16, 3, 3, Sum::Stages>;

// ---- skinny blocks (n, k ≤ 16): one thread per output row, op(B) in shared memory -----------
// Such blocks (tall-skinny GEMMs against small MPO bonds) are bound by reading op(A) and
// writing C; the row kernel streams both exactly once with coalesced accesses for op N.
template <typename T>
__device__ __forceinline__ T ldA(const T *p, bool conj);
template <>
__device__ __forceinline__ double ldA<double>(const double *p, bool) { return __ldg(p); }
template <>
__device__ __forceinline__ double2 ldA<double2>(const double2 *p, bool conj) {
  double2 v = __ldg(p);
  if (conj) v.y = -v.y;
  return v;
}
__device__ __forceinline__ double mac(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double2 mac(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
template <typename T>
__device__ __forceinline__ T make_beta(CDbl b);
template <>
__device__ __forceinline__ double make_beta<double>(CDbl b) { return b.x; }
template <>
__device__ __forceinline__ double2 make_beta<double2>(CDbl b) { return make_double2(b.x, b.y); }
__device__ __forceinline__ double zero(double) { return 0.0; }
__device__ __forceinline__ double2 zero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double scl(double v, CDbl a) { return a.x * v; }
__device__ __forceinline__ double2 scl(double2 v, CDbl a) {
  return make_double2(a.x * v.x - a.y * v.y, a.x * v.y + a.y * v.x);
}

// D bounds n and k of every block of the launch (2, 4, 6, 8 or 16). A CTA takes one task: the rows of
// one pass, R per thread. The R·k loads of op(A) are issued before op(B) is staged, so a thread
// keeps 8 - 16 values in flight (2 - 8 complex ones, with up to six CTAs per SM) while the CTA waits for
// op(B) as well.
// Blocks narrower than the launch's width class DK ≤ D take more rows per thread. Per element the
// arithmetic is acc = β·c (or 0), then acc = fma(α·a_l, op(B)_lj, acc) for l = 0 … k−1; rows where
// a_l was not loaded (invalid rows, l ≥ k) hold zeros and are not stored.
// Bound: HBM. 1.3 M rows of width 6: real 22 us (5.6 TB/s; 24 with persistent CTAs that staged op(B) before
// their loads and walked tasks of 1024 rows), ComplexF64 49 us (73 at three CTAs per SM); 580 K rows of
// width 12 31 us (41) and 82 us (135); 380 K rows of width 6 in ten blocks 6.1 us (8.0) and 10.5 us (16.3).
template <typename T, bool BZ, int D, int DK>
__device__ __forceinline__ void skinny_task(const GTile &tk, const GBlock &b, T *__restrict__ C, const T *__restrict__ A,
                                            const T *__restrict__ B, CDbl alpha, CDbl beta, T *Bs) {
  constexpr int RR = tkb_skinny_rows(sizeof(T) == 16, DK);
  const int n = (int)b.n, k = (int)b.k, kk = tk.kind == 0 ? k : 0;
  const int64_t m = b.m, ldc = b.ldc;
  const bool conjA = b.opA == TKB_OP_C;
  const int64_t sa_l = (b.opA == TKB_OP_N) ? b.lda : 1;
  const int64_t sa_i = (b.opA == TKB_OP_N) ? 1 : b.lda;
  const T *pa0 = A + b.offA;
  T *pc0 = C + b.offC;
  int64_t row[RR];
  bool valid[RR];
  T a[RR][DK];
#pragma unroll
  for (int r = 0; r < RR; ++r) {
    row[r] = (int64_t)tk.m0 + r * kSkinnyRows + threadIdx.x;
    valid[r] = row[r] < m;
  }
#pragma unroll
  for (int r = 0; r < RR; ++r)
#pragma unroll
    for (int l = 0; l < DK; ++l)
      a[r][l] = (valid[r] && l < kk) ? ldA<T>(pa0 + row[r] * sa_i + l * sa_l, conjA) : zero(T{});
  // op(B)(l, j), zero outside k × n
  for (int e = threadIdx.x; e < DK * DK; e += kSkinnyRows) {
    const int l = e % DK, j = e / DK;
    const int64_t idx = (b.opB == TKB_OP_N) ? b.offB + l + (int64_t)j * b.ldb : b.offB + j + (int64_t)l * b.ldb;
    Bs[e] = (l < kk && j < n) ? ldA<T>(B + idx, b.opB == TKB_OP_C) : zero(T{});
  }
  __syncthreads();
  // α·a once per element of op(A); each op(B)_lj is read from shared memory once
  // and used for the RR rows
#pragma unroll
  for (int r = 0; r < RR; ++r)
#pragma unroll
    for (int l = 0; l < DK; ++l) a[r][l] = scl(a[r][l], alpha);
#pragma unroll
  for (int j = 0; j < DK; ++j) {
    if (j < n) {
      T acc[RR];
#pragma unroll
      for (int r = 0; r < RR; ++r) {
        acc[r] = zero(T{});
        if constexpr (!BZ)
          if (valid[r]) acc[r] = mac(pc0[row[r] + (int64_t)j * ldc], make_beta<T>(beta), zero(T{}));
      }
#pragma unroll
      for (int l = 0; l < DK; ++l) {
        if (l < kk) {
          const T bl = Bs[l + j * DK];
#pragma unroll
          for (int r = 0; r < RR; ++r) acc[r] = mac(a[r][l], bl, acc[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < RR; ++r)
        if (valid[r]) pc0[row[r] + (int64_t)j * ldc] = acc[r];
    }
  }
}

// Resident CTAs asked of the register allocator: as many as fit without spills that cost more than
// the loads they add (the β ≠ 0 kernels also hold values of C)
template <typename T, bool BZ, int D>
constexpr int kSkinnyMinCtas = sizeof(T) == 8 ? (D <= 4 ? (BZ ? 6 : 4) : D == 6 ? (BZ ? 5 : 4) : D == 8 ? 4 : 2)
                                              : (D <= 4 ? (BZ ? 6 : 4) : D <= 8 ? (BZ ? 5 : 4) : BZ ? 3 : 2);

template <typename T, bool BZ, int D>
__global__ void __launch_bounds__(kSkinnyRows, kSkinnyMinCtas<T, BZ, D>)
    gemm_skinny_kernel(const GBlock *__restrict__ blocks, const GTile *__restrict__ tasks, T *__restrict__ C,
                       const T *__restrict__ A, const T *__restrict__ B, CDbl alpha, CDbl beta) {
  __shared__ T Bs[D * D];
  const GTile tk = tasks[blockIdx.x];
  const GBlock &b = blocks[tk.block];
  const int dk = tkb_skinny_class((int)b.n, (int)b.k);  // uniform over the CTA
  pdl_wait();
  pdl_trigger();
  if (D > 2 && dk == 2)
    skinny_task<T, BZ, D, 2>(tk, b, C, A, B, alpha, beta, Bs);
  else if (D > 4 && dk == 4)
    skinny_task<T, BZ, D, 4>(tk, b, C, A, B, alpha, beta, Bs);
  else
    skinny_task<T, BZ, D, D>(tk, b, C, A, B, alpha, beta, Bs);
}

}  // namespace

namespace {

template <typename T, bool BZ, int D>
int skinny_launch_t(tkb_ctx *ctx, const tkb_plan *p, T *C, const T *A, const T *B, CDbl a, CDbl bb) {
  TKB_CUDA_TRY(ctx, launch_pdl(gemm_skinny_kernel<T, BZ, D>, dim3((unsigned)p->nsk), dim3(kSkinnyRows), 0, ctx->stream,
                               p->blocks, p->sktasks, C, A, B, a, bb));
  return TKB_OK;
}

template <typename T, bool BZ>
int skinny_launch_d(tkb_ctx *ctx, const tkb_plan *p, T *C, const T *A, const T *B, CDbl a, CDbl bb) {
  const int d = p->sk_dim;
  if (d <= 2) return skinny_launch_t<T, BZ, 2>(ctx, p, C, A, B, a, bb);
  if (d <= 4) return skinny_launch_t<T, BZ, 4>(ctx, p, C, A, B, a, bb);
  if (d <= 6) return skinny_launch_t<T, BZ, 6>(ctx, p, C, A, B, a, bb);
  if (d <= 8) return skinny_launch_t<T, BZ, 8>(ctx, p, C, A, B, a, bb);
  return skinny_launch_t<T, BZ, 16>(ctx, p, C, A, B, a, bb);
}

}  // namespace

int tkb_gemm_skinny_launch(tkb_ctx *ctx, const tkb_plan *p, void *C, const void *A,
                           const void *B, tkb_scalar alpha, tkb_scalar beta) {
  if (p->nsk == 0) return TKB_OK;
  const CDbl a{alpha.re, alpha.im}, bb{beta.re, beta.im};
  const bool bz = beta.re == 0.0 && beta.im == 0.0;
  int rc;
  if (p->dtype == TKB_F64)
    rc = bz ? skinny_launch_d<double, true>(ctx, p, (double *)C, (const double *)A, (const double *)B, a, bb)
            : skinny_launch_d<double, false>(ctx, p, (double *)C, (const double *)A, (const double *)B, a, bb);
  else
    rc = bz ? skinny_launch_d<double2, true>(ctx, p, (double2 *)C, (const double2 *)A, (const double2 *)B, a, bb)
            : skinny_launch_d<double2, false>(ctx, p, (double2 *)C, (const double2 *)A, (const double2 *)B, a, bb);
  if (rc != TKB_OK) return rc;
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}

// ---- thin blocks (m, n ≤ 4, long K): a few dot products ----------------------------------------------
// Contractions that leave no legs open, or only a boundary of dimension 1 - 4, are dot products over
// K. A 64×64 tile does 1/4096 of its work on such a block and at most max_pieces CTAs share its K loop;
// here CTAs take K ranges, a thread keeps its loads of U·(m + n) values in flight, and the range that
// arrives last adds the ranges' sums in a fixed tree. Bound: HBM and, below a few MB, the launch. m = n = 1,
// K = 53764: 5.3 us real (158 tiled), 5.7 us ComplexF64 (1117); m = n = 4, K = 10⁶: 17 us real (2920), 115
// ComplexF64 with K contiguous (20550). The line at K = 512: 5.2 against 7.1 us real, 5.3 against
// 20.5 ComplexF64 for a block alone; shorter blocks are not worth a launch of their own beside a tiled one.
namespace {

__device__ __forceinline__ double shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double2 shfl_xor(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ double plus(double a, double b) { return a + b; }
__device__ __forceinline__ double2 plus(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double ldcg_v(const double *p) { return __ldcg(p); }
__device__ __forceinline__ double2 ldcg_v(const double2 *p) { return __ldcg(p); }

constexpr int kThinThreads = 256;

template <typename T, int D>
__global__ void __launch_bounds__(kThinThreads)
    gemm_thin_kernel(const GBlock *__restrict__ blocks, const ThinTask *__restrict__ tasks, T *__restrict__ C,
                     const T *__restrict__ A, const T *__restrict__ B, CDbl alpha, CDbl beta, T *__restrict__ part,
                     int *__restrict__ cnt) {
  constexpr int DD = D * D, U = D == 1 ? 4 : D == 2 ? 2 : 1;
  __shared__ T red[kThinThreads / 32][DD];
  __shared__ int last;
  const ThinTask t = tasks[blockIdx.x];
  const GBlock &b = blocks[t.block];
  const int m = (int)b.m, n = (int)b.n;
  const int64_t ai = b.opA == TKB_OP_N ? 1 : b.lda, al = b.opA == TKB_OP_N ? b.lda : 1;
  const int64_t bj = b.opB == TKB_OP_N ? b.ldb : 1, bl = b.opB == TKB_OP_N ? 1 : b.ldb;
  const bool ca = b.opA == TKB_OP_C, cb = b.opB == TKB_OP_C;
  const T *pa = A + b.offA, *pb = B + b.offB;
  pdl_wait();
  pdl_trigger();
  T acc[DD];
#pragma unroll
  for (int e = 0; e < DD; ++e) acc[e] = zero(T{});
  for (int64_t l0 = t.l0 + threadIdx.x; l0 < t.l1; l0 += kThinThreads * U) {
    T a[U][D], v[U][D];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t l = l0 + u * kThinThreads;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        a[u][i] = l < t.l1 && i < m ? ldA<T>(pa + i * ai + l * al, ca) : zero(T{});
        v[u][i] = l < t.l1 && i < n ? ldA<T>(pb + i * bj + l * bl, cb) : zero(T{});
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < D; ++j)
#pragma unroll
        for (int i = 0; i < D; ++i)
          if (i < m && j < n && l0 + u * kThinThreads < t.l1) acc[i + j * D] = mac(a[u][i], v[u][j], acc[i + j * D]);
  }
  // sum over the CTA: thread e < DD holds value e
  auto total = [&]() {
#pragma unroll
    for (int e = 0; e < DD; ++e)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[e] = plus(acc[e], shfl_xor(acc[e], o));
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int e = 0; e < DD; ++e) red[threadIdx.x >> 5][e] = acc[e];
    }
    __syncthreads();
    T s = zero(T{});
    if (threadIdx.x < DD)
      for (int w = 0; w < kThinThreads / 32; ++w) s = plus(s, red[w][threadIdx.x]);
    __syncthreads();
    return s;
  };
  T sum = total();
  if (t.nsplit > 1) {
    if (threadIdx.x < DD) part[(int64_t)(t.pbase + t.sid) * DD + threadIdx.x] = sum;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&cnt[t.slot], 1) == t.nsplit - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int e = 0; e < DD; ++e) acc[e] = zero(T{});
    for (int sp = threadIdx.x; sp < t.nsplit; sp += kThinThreads)
#pragma unroll
      for (int e = 0; e < DD; ++e) acc[e] = plus(acc[e], ldcg_v(&part[(int64_t)(t.pbase + sp) * DD + e]));
    sum = total();
    if (threadIdx.x == 0) cnt[t.slot] = 0;  // every range has arrived
  }
  const int i = threadIdx.x % D, j = threadIdx.x / D;
  if (threadIdx.x < DD && i < m && j < n) {
    T *p = C + b.offC + i + j * b.ldc;
    T r = scl(sum, alpha);
    if (beta.x != 0.0 || beta.y != 0.0) r = mac(make_beta<T>(beta), *p, r);
    *p = r;
  }
}

template <typename T>
cudaError_t thin_launch(tkb_ctx *ctx, const tkb_plan *p, void *C, const void *A, const void *B, CDbl a, CDbl b) {
  auto k = p->th_dim <= 1 ? gemm_thin_kernel<T, 1> : p->th_dim <= 2 ? gemm_thin_kernel<T, 2> : gemm_thin_kernel<T, 4>;
  return launch_pdl(k, dim3((int)p->nth), dim3(kThinThreads), 0, ctx->stream, p->blocks, p->thtasks, (T *)C,
                    (const T *)A, (const T *)B, a, b, (T *)p->thpart, p->thcnt);
}

}  // namespace

int tkb_gemm_thin_launch(tkb_ctx *ctx, const tkb_plan *p, void *C, const void *A, const void *B,
                         tkb_scalar alpha, tkb_scalar beta) {
  if (p->nth == 0) return TKB_OK;
  if (p->dtype == TKB_F64 && (alpha.im != 0.0 || beta.im != 0.0))
    return tkb_set_error(ctx, TKB_ERR_ARG, "complex scalar with real data");
  if (p->dtype == TKB_C128 && (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) != 0)
    return tkb_set_error(ctx, TKB_ERR_ARG, "ComplexF64 data must be 16-byte aligned");
  const CDbl a{alpha.re, alpha.im}, b{beta.re, beta.im};
  TKB_CUDA_TRY(ctx, p->dtype == TKB_F64 ? thin_launch<double>(ctx, p, C, A, B, a, b)
                                        : thin_launch<double2>(ctx, p, C, A, B, a, b));
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}

// Work decomposition of a plain GEMM: the tile shape and the tasks of every CTA.
// - Real: LargeTile runs where its tiles, cut in K as far as they may be, fill the chip (at least 0.85 pieces
//   per resident CTA) and padding to it costs at most a fifth more K steps than padding to SmallTile. us, large /
//   small: one 60x2400x2400 block (304 pieces) 37 / 45, 120x1200x1200 24 / 27, 1000x20x1000 (256) 7.0 / 9.4,
//   512x100x512 (128) 11.9 / 7.6, 200x5000x100 (64) 46 / 29, 30 blocks of 70 (1.8 times the steps) 11.1 / 6.5,
//   heff of V dim 750 (1.23 times) 21.5 / 19.8, 6 blocks of 300 27 / 25.
// - Complex: SmallTileC runs up to 16 tiles per SM, LargeTileC above (2048^3: 30.6 and 32.7 TFLOP/s). Between 6 and 16
//   tiles per SM the large one is up to a tenth faster, but it has one accumulator and fewer pieces of K.
// - Fewer tiles than resident CTAs: the K loops of the longest tiles are cut into equal pieces of the
//   shortest length (at least min_piece_steps K steps) whose count still fits, one task per CTA.
// - Otherwise, and where those pieces would leave a tenth of the CTAs or more without one although the work is long
//   (24 steps of the small tile for everyone) and the tiles may be cut fine enough, every CTA gets an equal share of
//   all K steps (plus tile_cost steps per tile for its
//   epilogue), as a contiguous range of the tiles in order of falling K; a tile that a share ends in
//   is cut there. Whole tiles alone leave CTAs idle for up to a tile each: on a U(1) effective
//   Hamiltonian's second product (394 tiles of up to 109 steps for 296 CTAs) SMs were active for
//   70 % of the launch. A CTA runs its cut tiles first, so their partial sums meet while it goes on. One complex
//   60x2400x2400 block (300 equal pieces for 444 CTAs) takes 112 us in shares and 158 in pieces, 257x1736x400 67 and
//   80; shorter work loses (512^3 48 and 44, 18 steps each; ten blocks of 150 22 and 17, 6 steps each).

namespace {
struct PlainKernel {
  const void *fn, *fn_beta;  // without and with β
  int threads, bm, bn;
  size_t smem;
};
template <typename CFG>
PlainKernel plain_kernel_of() {
  return PlainKernel{(const void *)gemm_plain_kernel<CFG, CFG::BETA_KERNEL>, (const void *)gemm_plain_kernel<CFG, false>, CFG::THREADS,
                     CFG::BM, CFG::BN, CFG::SMEM};
}
// CTAs per SM of both kernels of a shape (raises their shared memory limits)
int plain_occupancy(tkb_ctx *ctx, const PlainKernel &k) {
  return std::min(tkb_occupancy(ctx->device, k.fn, k.threads, k.smem),
                  tkb_occupancy(ctx->device, k.fn_beta, k.threads, k.smem));
}
PlainKernel plain_kernel(bool cplx, bool small) {
  return cplx ? (small ? plain_kernel_of<SmallTileC>() : plain_kernel_of<LargeTileC>())
              : (small ? plain_kernel_of<SmallTile>() : plain_kernel_of<LargeTile>());
}
template <typename CFG>
cudaError_t plain_launch(tkb_ctx *ctx, const tkb_plan *p, void *C, const void *A, const void *B, tkb_scalar alpha,
                         tkb_scalar beta, int base_ok) {
  using E = typename CFG::E;
  // the shared-memory limit was raised when the plan queried the kernel's occupancy
  const auto k = beta.re == 0.0 && beta.im == 0.0 ? gemm_plain_kernel<CFG, CFG::BETA_KERNEL> : gemm_plain_kernel<CFG, false>;
  return launch_pdl(k, dim3(p->pgrid), dim3(CFG::THREADS), CFG::SMEM, ctx->stream, p->blocks,
                    (const PTask *)p->ptasks, (const int32_t *)p->pstart, (E *)C, (const E *)A, (const E *)B,
                    CDbl{alpha.re, alpha.im}, CDbl{beta.re, beta.im}, p->part, p->pcnt, base_ok);
}
}  // namespace

int tkb_gemm_plain_prepare(tkb_ctx *ctx, tkb_plan *p) {
  const bool cplx = p->dtype == TKB_C128;
  auto tiles_of = [](const GBlock &b, const PlainKernel &k) { return ((b.m + k.bm - 1) / k.bm) * ((b.n + k.bn - 1) / k.bn); };
  const PlainKernel large = plain_kernel(cplx, false), small = plain_kernel(cplx, true);
  int64_t small_tiles = 0, small_steps = 0, large_steps = 0, large_pieces = 0;
  for (const GBlock &b : p->hblocks) {
    if (b.skinny) continue;
    const int64_t nk = (b.k + BK - 1) / BK, tl = tiles_of(b, large), ts = tiles_of(b, small);
    small_tiles += ts;
    small_steps += ts * nk;
    large_steps += tl * nk;
    large_pieces += tl * std::min<int64_t>(p->max_pieces, std::max<int64_t>(1, (nk + p->min_piece_steps - 1) / p->min_piece_steps));
  }
  if (cplx) {
    p->plain_small = small_tiles <= (int64_t)ctx->num_sms * 16;
  } else {
    const int large_sm = plain_occupancy(ctx, large);
    const bool fills = large_pieces * 20 >= (int64_t)ctx->num_sms * large_sm * 17;
    const bool padded = large_steps * 4 * 5 > small_steps * 6;  // a step of the large tile is four of the small one
    p->plain_small = !fills || padded;
  }
  const PlainKernel pk = plain_kernel(cplx, p->plain_small);
  const int tm = pk.bm, tn = pk.bn;
  // a piece's partial sums cost as much as twice as many steps of the smaller tile; a complex step is
  // four real ones
  const int min_steps = std::max(1, p->min_piece_steps * (p->plain_small ? 2 : 1) / (cplx ? 4 : 1));
  const int tile_cost = cplx ? 1 : 2;
  const int per_sm = plain_occupancy(ctx, pk);
  if (per_sm <= 0) return tkb_set_error(ctx, TKB_ERR_CUDA, "plain GEMM: occupancy query failed");
  const int64_t slots = (int64_t)ctx->num_sms * per_sm;
  std::vector<GTile> tiles;
  for (size_t i = 0; i < p->hblocks.size(); ++i) {
    const GBlock &b = p->hblocks[i];
    if (b.skinny) continue;
    for (int64_t m0 = 0; m0 < b.m; m0 += tm)
      for (int64_t n0 = 0; n0 < b.n; n0 += tn)
        tiles.push_back({(int32_t)i, (int32_t)m0, (int32_t)n0, b.k > 0 ? 0 : 1});
  }
  std::stable_sort(tiles.begin(), tiles.end(),
                   [&](const GTile &x, const GTile &y) { return p->hblocks[x.block].k > p->hblocks[y.block].k; });
  const int64_t nt = (int64_t)tiles.size();
  int64_t total = 0, maxnk = 1;
  std::vector<int64_t> nks(nt);
  for (int64_t i = 0; i < nt; ++i) {
    const GTile &t = tiles[i];
    nks[i] = t.kind == 0 ? (p->hblocks[t.block].k + BK - 1) / BK : 0;
    total += nks[i];
    maxnk = std::max(maxnk, nks[i]);
  }
  std::vector<std::vector<PTask>> lists;  // per CTA
  int nslots = 0, npart = 0;
  auto pieces = [&](int64_t nk, int64_t target) {
    return (int)std::min<int64_t>(p->max_pieces, std::max<int64_t>(1, (nk + target - 1) / target));
  };
  int64_t target = std::max<int64_t>(min_steps, (total + slots - 1) / slots), cnt = nt;
  if (nt < slots) {
    for (;; ++target) {
      cnt = 0;
      for (int64_t i = 0; i < nt; ++i) cnt += pieces(nks[i], target);
      if (cnt <= slots || target >= maxnk) break;
    }
  }
  const bool shares = nt >= slots || (cnt * 10 < slots * 9 && nt * p->max_pieces * 2 >= slots * 3 &&
                                      total >= slots * (p->plain_small ? 24 : 12));
  if (!shares) {
    for (int64_t i = 0; i < nt; ++i) {
      const GTile &t = tiles[i];
      const int nk = (int)nks[i];
      const int ks = t.kind == 0 ? pieces(nk, target) : 1;
      const int slot = ks > 1 ? nslots++ : -1;
      for (int s = 0; s < ks; ++s)
        lists.push_back({PTask{t.block, t.m0, t.n0, t.kind, (int32_t)((int64_t)s * nk / ks),
                               (int32_t)((int64_t)(s + 1) * nk / ks), slot, ks, s, ks > 1 ? npart : 0}});
      if (ks > 1) npart += ks;
    }
    std::stable_sort(lists.begin(), lists.end(), [](const std::vector<PTask> &x, const std::vector<PTask> &y) {
      return x[0].ke - x[0].kb > y[0].ke - y[0].kb;
    });
  } else {
    lists.resize((size_t)slots);
    std::vector<std::vector<PTask>> whole((size_t)slots);
    const double share = (double)(total + tile_cost * nt) / (double)slots;
    double pos = 0.0;  // steps given out so far
    int64_t cta = 0;
    for (int64_t i = 0; i < nt; ++i) {
      const GTile &t = tiles[i];
      int64_t kb = 0;
      std::vector<std::pair<int64_t, PTask>> cut;  // (CTA, piece)
      while (true) {
        const int64_t len = nks[i] - kb;
        while (cta + 1 < slots && pos >= share * (double)(cta + 1)) ++cta;
        const double room = share * (double)(cta + 1) - pos;
        int64_t head = (int64_t)room;  // steps of this piece that fit the CTA's share
        const bool may_cut = cta + 1 < slots && (int64_t)cut.size() + 1 < p->max_pieces;
        if (!may_cut || len - head < min_steps) {
          head = len;  // the rest of the tile, where what would be left over is not worth a piece
        } else if (head < min_steps) {
          ++cta;       // the share ends here
          continue;
        }
        cut.push_back({cta, PTask{t.block, t.m0, t.n0, t.kind, (int32_t)kb, (int32_t)(kb + head), -1, 1, 0, 0}});
        kb += head;
        pos += (double)head;
        if (kb >= nks[i]) break;
      }
      pos += tile_cost;
      const int ks = (int)cut.size();
      if (ks == 1) {
        whole[cut[0].first].push_back(cut[0].second);
        continue;
      }
      for (int s = 0; s < ks; ++s) {
        PTask q = cut[s].second;
        q.slot = nslots;
        q.nsplit = ks;
        q.sid = s;
        q.pbase = npart;
        lists[cut[s].first].push_back(q);
      }
      ++nslots;
      npart += ks;
    }
    for (int64_t c = 0; c < slots; ++c) lists[c].insert(lists[c].end(), whole[c].begin(), whole[c].end());
    lists.erase(std::remove_if(lists.begin(), lists.end(), [](const std::vector<PTask> &l) { return l.empty(); }),
                lists.end());
  }
  std::vector<PTask> tasks;
  std::vector<int32_t> start{0};
  for (const auto &l : lists) {
    tasks.insert(tasks.end(), l.begin(), l.end());
    start.push_back((int32_t)tasks.size());
  }
  p->nptasks = (int64_t)tasks.size();
  p->pgrid = (int)lists.size();
  cudaError_t e = cudaSuccess;
  if (!tasks.empty()) {
    e = cudaMalloc(&p->ptasks, tasks.size() * sizeof(PTask));
    if (e == cudaSuccess) e = cudaMemcpy(p->ptasks, tasks.data(), tasks.size() * sizeof(PTask), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc((void **)&p->pstart, start.size() * sizeof(int32_t));
    if (e == cudaSuccess)
      e = cudaMemcpy(p->pstart, start.data(), start.size() * sizeof(int32_t), cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess && nslots > 0) {
    e = cudaMalloc((void **)&p->part, (size_t)npart * tm * tn * (cplx ? 2 : 1) * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc((void **)&p->pcnt, nslots * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(p->pcnt, 0, nslots * sizeof(int));
  }
  if (e != cudaSuccess)
    return tkb_set_error(ctx, TKB_ERR_CUDA, std::string("plain plan upload: ") + cudaGetErrorString(e));
  return TKB_OK;
}

int tkb_gemm_launch(tkb_ctx *ctx, const tkb_plan *p, void *C, const void *A, const void *B,
                    tkb_scalar alpha, tkb_scalar beta) {
  if (p->nptasks == 0) return TKB_OK;
  if (p->dtype == TKB_F64) {
    if (alpha.im != 0.0 || beta.im != 0.0)
      return tkb_set_error(ctx, TKB_ERR_ARG, "complex scalar with real data");
    const int base_ok = (((uintptr_t)A & 15) == 0 ? 1 : 0) | (((uintptr_t)B & 15) == 0 ? 2 : 0);
    TKB_CUDA_TRY(ctx, p->plain_small ? plain_launch<SmallTile>(ctx, p, C, A, B, alpha, beta, base_ok)
                                     : plain_launch<LargeTile>(ctx, p, C, A, B, alpha, beta, base_ok));
  } else {
    if ((((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) != 0)
      return tkb_set_error(ctx, TKB_ERR_ARG, "ComplexF64 data must be 16-byte aligned");
    TKB_CUDA_TRY(ctx, p->plain_small ? plain_launch<SmallTileC>(ctx, p, C, A, B, alpha, beta, 0)
                                     : plain_launch<LargeTileC>(ctx, p, C, A, B, alpha, beta, 0));
  }
  ctx->launches++;
  TKB_CUDA_TRY(ctx, cudaGetLastError());
  return TKB_OK;
}

#ifdef TKB_TIMELINE
// copies the plain kernel's per-CTA stamps out (kPlTlCtas × kPlTlSlots values) and clears them
extern "C" int tkb_timeline_read_plain(unsigned long long *out) {
  if (cudaMemcpyFromSymbol(out, tkb_tl_plain, sizeof(tkb_tl_plain)) != cudaSuccess) return -1;
  static unsigned long long zero[kPlTlCtas * kPlTlSlots];
  return cudaMemcpyToSymbol(tkb_tl_plain, zero, sizeof(tkb_tl_plain)) == cudaSuccess ? kPlTlSlots : -1;
}
#endif
