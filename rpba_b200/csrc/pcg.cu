// pcg.cu -- block-Jacobi preconditioned conjugate gradients on the reduced
// camera system, with the scalar logic of SparsePCG (rbacore.cpp:1807-1914):
// x0 = 0, best iterate kept (starting from the right-hand side), stop when
// the squared step increment drops by 1e5 or after msize iterations,
// beta = r1^T (h1 - h) / r^T h clamped at 0.
//
// One cooperative launch runs the whole solve.  The FP64 form is k_pcg, the
// FP32 form k_pcg32; each has a variant for systems that stay in shared memory
// (described before them).  Dot products are reduced per CTA and then, after a
// grid barrier, by every CTA in the same fixed order, so all CTAs take
// identical decisions.  The grid barrier's wait is bounded: after 2 s it sets
// an error bit and returns.
#include <cooperative_groups.h>

#include <algorithm>

#include "gridsync.cuh"
#include "internal.h"

namespace rpba {

namespace {

// Threads and warps per CTA of the FP64 form's persistent kernel.
constexpr int P64_T = 1024, P64_W = P64_T / 32;

struct PcgArgs {
  const void *blocks;  // [(nimg + nboff) * 81] doubles or floats
  const int *row_item_off;
  const int2 *item_rec;   // [nitems][4 or 1] (row | entries << 16, first entry), resident form: up to three entries
  const int2 *ent;        // gathered form: the entries
  double *prod;           // FP64 streamed form: the product of every entry, 9 values each, entry order
  float *tpart;           // FP32 form: transposed products of the off-diagonal blocks
  // (row, column) of every block in storage order, with its transposed slot
  // (FP32 form) or its two entries (FP64 form: normal, transposed); the
  // first off-diagonal block of every row, d^k in FP32 (12 floats a camera),
  // and the phase-1 row sums (diagonal, row head, warp-run head)
  const int4 *bidx;
  const int *firstN, *firstT;
  int nboff;
  float *d32;
  double *pdiag, *prow, *pw;  // pw: per chunk
  double *pdqc;               // per chunk: its share of d^T A d
  unsigned *ctr;              // next chunk of phase 1
  int chunk;                  // groups per phase-1 chunk
  int g0;                     // CTAs whose rows' sums are added (SMALL)
  const double *Cinv;
  double *r, *h, *x, *xbest, *D0, *D1;
  double *part;        // [nitems * 9] SpMV partial rows
  // per-CTA sums of phase 1 and of phase 2, [N][XMAXG] (separate, so a fast
  // CTA never overwrites a slot that a slow CTA is still reading)
  double *red1, *red2;
  unsigned *bar;       // [0]: GridBarrier, [1]: the exchanges
  int *err;
  int *iters;
  // grid barriers wait for G + bar_extra arrivals, at most bar_ns each
  // (bar_extra 0 and the default limit outside the timeout test hook)
  unsigned bar_extra;
  unsigned long long bar_ns;
  unsigned tx_extra;
  int row0, row1, nitems, msize;
  int stream_once;  // FP64 streamed form: blocks read with an evict-first hint
  int mode;     // 0: reference stop rule; 1: relative preconditioned residual
  double tol2;  // mode 1: stop when r^T M^-1 r <= tol2 * (r0^T M^-1 r0)
  // two-level preconditioner (coarse.cu): rows are owned per aggregate
  int nagg, nc;
  const int *agg_off, *agg_rows;
  const double *P, *Ainv;
  double *rc, *hj;
  double *rowc;  // FP32 form: per row its restriction P_k^T r1 (CO_M) and its share of dr^2, stride RC_S
};

// Sum of N values over the CTAs with the barrier between the phases in it:
// each CTA's sum is stored, all CTAs arrive and wait, and every CTA reads all
// the sums.  All writes a CTA made before the call are visible to all CTAs
// after it.  The order of the additions is fixed: lanes of a warp
// (butterfly), warps (butterfly over the W warps' sums), CTAs (lane l takes
// l, l + 32, ...; butterfly), so every CTA gets the same values.  Bounded like
// GridBarrier's wait, and `bad` as there: false in every thread when it ran
// out or a thread of the CTA passed bad.  (Every CTA
// polling the others' tagged sums themselves instead saves the read, but 148
// CTAs polling 148 slots took 14,000 cycles where this takes 5,000.)
constexpr int XMAXG = 256;  // CTAs at most
template <int N, int W>
struct Exchange {
  double warp[W][N];
  double cta[XMAXG * N];
};
template <int N, int W>
__device__ __forceinline__ bool exchange_sum(GridBarrier &bar, double *red, double (&v)[N], Exchange<N, W> &X,
                                             int bad = 0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < N; ++j) X.warp[warp][j] = v[j];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
      double t = lane < W ? X.warp[lane][j] : 0.;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) red[j * XMAXG + blockIdx.x] = t;
    }
  }
  // (thread 0 wrote the CTA's sums; every other write of the CTA came before
  // the block barrier above)
  if (!bar.sync_after_block(bad)) return false;
  if (threadIdx.x < G)
#pragma unroll
    for (int j = 0; j < N; ++j) X.cta[j * XMAXG + threadIdx.x] = __ldcg(red + j * XMAXG + threadIdx.x);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; ++j) {
    double t = 0.;
    for (int i = lane; i < G; i += 32) t += X.cta[j * XMAXG + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    v[j] = t;
  }
  return true;
}

// ---- mbarriers and bulk copies (1-D TMA, one destination CTA)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// global -> shared bulk copy completing on `bar` (one destination: this
// CTA's own shared memory; the source is this GPU's own memory)
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// the same with an L2 policy; policy 0: none
__device__ __forceinline__ void bulk_load_hint(void *dst, const void *src, unsigned bytes, unsigned long long *bar,
                                               unsigned long long policy) {
  if (policy == 0) {
    bulk_load(dst, src, bytes, bar);
    return;
  }
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// Bounded wait of a whole warp on the stage's mbarrier (the copies of this
// CTA's own memory end in microseconds; the limit only keeps a fault from
// hanging): one result for all lanes.
__device__ __forceinline__ bool stage_wait(const PcgArgs &A, unsigned long long *bar, unsigned parity) {
  bool ok = mbar_try_wait(bar, parity);
  if (!ok) {
    const unsigned long long t0 = gtimer();
    while (!(ok = mbar_try_wait(bar, parity)))
      if (gtimer() - t0 > A.bar_ns) break;
  }
  return __all_sync(0xffffffffu, ok);
}
// bytes that no copy brings, added to what the stages of CTA 0 expect (0
// outside the test hook)
__device__ __forceinline__ unsigned tx_extra(const PcgArgs &A) { return blockIdx.x == 0 ? A.tx_extra : 0u; }

// Phase 1 of the FP64 form: q-partials p = sum of B d^k over the (at most
// three) entries of every work item, and d^T A d.  A warp's items (gwarp,
// gwarp + nwarps, ...) are the same in every iteration, and so are the
// blocks.  Three forms with the same operations in the same order per entry
// and per item:
//  resident   at most P1_SLOTS items a warp: their blocks and records stay in
//             shared memory for the whole solve; a 9-lane group forms each
//             entry's product and the warp the item's sum.
//  streamed   more: phase 1a reads every block once, in storage order, by
//             1-D TMA bulk copies of 32 blocks into P1S_N stages a CTA (a
//             stage with one group keeps it for the whole solve); two warps
//             a stage, a lane a block, form B d_col and B^T d_row and store
//             them at their entries' places (vectors copied in and products
//             written through shared memory in whole 72-byte pieces); a grid
//             barrier; phase 1b sums every item's products.  Half the block
//             traffic of reading each block from both sides, in copies of
//             20 KB, for one more barrier.
//  gathered   the resident form's sums with the blocks read from global
//             memory in every iteration, from both sides: needs no memory for
//             products, taken only where there is none.
// The threads have 64 registers each and the stages leave L1 some 20 KB, so
// spilled registers cost L2 trips: a spill of 50 to 100 bytes was worth 10 to
// 30%.  Iteration, before (each block read from both sides, 8-byte copies two
// items ahead, the records through two dependent loads) and now: 50 cameras
// 14.0 -> 10.0 us (resident), 3,000 cameras and 27,000 blocks 24.0 -> 17.3 us,
// 1,370 cameras and 371,000 blocks 137 -> 115 us (streamed).
constexpr int P1_SLOTS = 3;
constexpr unsigned P1_PIECE = 656;  // a block's 648 bytes from the 16-byte boundary at or below it
constexpr unsigned P1_WARP_BYTES = P1_SLOTS * (3 * P1_PIECE + 32) + 648 + 8;  // blocks, records, C of a row, mbarrier
static_assert(P1_WARP_BYTES % 16 == 0, "16-byte aligned pieces");
constexpr int P1S_N = 7;                                  // stages per CTA (two warps each)
constexpr unsigned P1S_BLK = 32 * 648 + 16;               // a group's blocks
constexpr unsigned P1S_IDX = 32 * 16;                     // and their indices
constexpr unsigned P1S_BUF = 32 * 9 * 8;                  // a warp's 32 h or d^(k-1), or products
constexpr unsigned P1S_STAGE = P1S_BLK + P1S_IDX + 4 * P1S_BUF + 16;  // + the mbarrier
static_assert(P1S_BLK % 16 == 0 && P1S_STAGE % 16 == 0, "16-byte aligned stage parts");
template <int FORM>
constexpr size_t pcg_smem_bytes() {
  return FORM == PCG_STREAMED ? (size_t)P1S_N * P1S_STAGE
                              : (FORM == PCG_RESIDENT ? (size_t)P64_W * P1_WARP_BYTES : 0);
}

__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Groups of 32 blocks in storage order: the diagonal blocks of the system's
// rows, then the off-diagonal blocks.
struct Grp64 {
  long long start;
  int n;
  bool diag;
};
__device__ __forceinline__ Grp64 group64(const PcgArgs &A, int g) {
  const int gd = (A.row1 - A.row0 + 31) / 32;
  Grp64 q;
  if (g < gd) {
    q.start = A.row0 + 32ll * g;
    q.n = (int)min(32ll, A.row1 - q.start);
    q.diag = true;
  } else {
    const long long o = 32ll * (g - gd);
    q.start = A.row1 + o;
    q.n = (int)min(32ll, A.nboff - o);
    q.diag = false;
  }
  return q;
}
__device__ __forceinline__ void group64_issue(const PcgArgs &A, int g, unsigned char *stg, unsigned long long *mbar,
                                              unsigned long long policy) {
  const Grp64 q = group64(A, g);
  const unsigned long long src = (unsigned long long)A.blocks + (unsigned long long)q.start * 648u;
  const unsigned mis = (unsigned)(src & 15ull), nb = (mis + (unsigned)q.n * 648u + 15u) & ~15u;
  mbar_expect_tx(mbar, nb + (unsigned)q.n * 16u + tx_extra(A));
  bulk_load_hint(stg, (const void *)(src - mis), nb, mbar, policy);
  bulk_load(stg + P1S_BLK, A.bidx + q.start, (unsigned)q.n * 16u, mbar);
}

// q of one row (valid in lanes < 9) from the phase-1 partials of the FP64
// form: one partial per item, the three 9-lane groups taking every third
// item, in a fixed order (four running sums of a group, items t, t + 3, t + 6,
// t + 9 of every twelve; the last, incomplete twelve onto the first sum); the
// loads of two twelves are in flight before they are added.
__device__ __forceinline__ double row_q(const PcgArgs &A, int t0, int t1, int lane, int grp, int rr) {
  double qg = 0.;
  if (lane < 27) {
    double q0 = 0., q1 = 0., q2 = 0., q3 = 0.;
    int t = t0 + grp;
    const double *p = A.part + rr;
#pragma unroll 2
    for (; t + 9 < t1; t += 12) {
      double u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = __ldcg(p + (size_t)(t + 3 * j) * 9);
      q0 += u[0];
      q1 += u[1];
      q2 += u[2];
      q3 += u[3];
    }
    double u[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) u[j] = t + 3 * j < t1 ? __ldcg(p + (size_t)(t + 3 * j) * 9) : 0.;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (t + 3 * j < t1) q0 += u[j];
    qg = (q0 + q1) + (q2 + q3);
  }
  const double qa = __shfl_down_sync(0xffffffffu, qg, 9);
  const double qb = __shfl_down_sync(0xffffffffu, qg, 18);
  return qg + qa + qb;
}

// Iteration k (two grid barriers, three in the streamed form):
//  phase 1  q-partials of A d^k per work item (<= 3 blocks of one row), with
//           d^k = h^k + beta^(k-1) d^(k-1) formed on the fly; partial d^T q
//  phase 2  per row: q = sum of its items' partials, x += alpha d,
//           r1 = r - alpha q, h1 = C r1; partials of (alpha q)^2,
//           r1^T (h1 - h) and r1^T h1 (the next r^T h); d^k is stored
// With the coarse correction (CO) phase 2 is split by one more barrier:
//  phase 2a per aggregate (one CTA): as above but h1 is only the block part
//           (kept in hj), and the aggregate's restriction P^T r1 is formed
//  phase 2b per aggregate: z = A_c^-1[aggregate rows] (P^T r1), then
//           h1 = hj + P z and the two dot products
template <bool CO, int FORM>
__global__ void __launch_bounds__(P64_T, 1) k_pcg(PcgArgs A) {
  constexpr bool RES = FORM == PCG_RESIDENT, SYM = FORM == PCG_STREAMED;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = blockIdx.x * P64_W + warp, nwarps = gridDim.x * P64_W;
  const int grp = lane / 9, rr = lane % 9, gbase = grp * 9;
  const int G = gridDim.x;
  GridBarrier bar(A.bar, (unsigned)G + A.bar_extra, A.err, A.bar_ns);
  __shared__ Exchange<1, P64_W> X1;
  __shared__ Exchange<3, P64_W> X2;
  // scalars of the recurrence by iteration parity (every thread computes the
  // same values, thread 0 stores them): r^T h, its start value, the smallest
  // and the first increment
  __shared__ double sc[2][4];
  extern __shared__ __align__(16) unsigned char pcg_dyn[];
  // this warp's items
  const int T = gwarp < A.nitems ? (A.nitems - 1 - gwarp) / nwarps + 1 : 0;
  // resident form: blocks, records, C of the warp's first row, mbarrier;
  // streamed form: a stream warp's stage and its groups gs, gs + gstep, ...
  unsigned char *stg = pcg_dyn + (SYM ? (size_t)(warp >> 1) * P1S_STAGE : (size_t)warp * P1_WARP_BYTES);
  int2 *recs = (int2 *)(stg + P1_SLOTS * 3 * P1_PIECE);
  double *Cs = (double *)(recs + 4 * P1_SLOTS);
  unsigned long long *mbar =
      SYM ? (unsigned long long *)(stg + P1S_STAGE - 16) : (unsigned long long *)(Cs + 81);
  const int ng = (A.row1 - A.row0 + 31) / 32 + (A.nboff + 31) / 32;
  const int gs = (warp >> 1) * G + (int)blockIdx.x, gstep = P1S_N * G;
  const bool stream = SYM && warp < 2 * P1S_N && gs < ng;
  const bool keep = ng <= gstep;  // every stage's only group stays
  unsigned parity = 0;
  // false: a copy that never completed (bounded wait); nothing is taken from
  // its stage, no other copy is issued to it, and the CTA leaves at the next
  // grid barrier
  bool ok = true;
  unsigned long long policy = 0;
  if constexpr (SYM) {
    if (stream) {
      // blocks that do not fit L2 beside the products should not evict them
      // (STREAM_ONCE_BYTES)
      if (A.stream_once)
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(policy));
      if (lane == 0 && (warp & 1) == 0) {
        mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        group64_issue(A, gs, stg, mbar, policy);
      }
    }
    __syncthreads();  // the mbarriers are initialised
  } else if constexpr (RES) {
    if (lane < 4 * T) recs[lane] = __ldg(A.item_rec + 4 * ((size_t)gwarp + (size_t)(lane >> 2) * nwarps) + (lane & 3));
    __syncwarp();
    if (lane == 0 && T > 0) {
      mbar_init(mbar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
      int np = 0;
      for (int t = 0; t < T; ++t) np += recs[4 * t].x >> 16;
      mbar_expect_tx(mbar, (unsigned)np * P1_PIECE + tx_extra(A));
      for (int t = 0; t < T; ++t)
        for (int g = 0; g < (recs[4 * t].x >> 16); ++g)
          bulk_load(stg + (3 * t + g) * P1_PIECE,
                    (const unsigned char *)A.blocks +
                        (((size_t)(recs[4 * t + 1 + g].y & 0x7fffffff) * 648u) & ~(size_t)15),
                    P1_PIECE, mbar);
    }
    __syncwarp();
  }
  // the copies in flight end before the CTA does
  bool landed = false;
  auto drain = [&]() {
    if (SYM ? stream : (RES && T > 0 && !landed)) stage_wait(A, mbar, parity);
  };
  // the warp's first row of phase 2: its items and preconditioner block
  const int rowa = A.row0 + gwarp;
  const bool has_row = !CO && rowa < A.row1;
  const int ta0 = has_row ? A.row_item_off[rowa] : 0, ta1 = has_row ? A.row_item_off[rowa + 1] : 0;
  if (RES && has_row)
    for (int e = lane; e < 81; e += 32) Cs[e] = __ldg(A.Cinv + (size_t)rowa * 81 + e);
  // r^T h of the start vectors
  {
    double v[3] = {0., 0., 0.};
    for (int row = A.row0 + gwarp; row < A.row1; row += nwarps)
      if (lane < 9) {
        const size_t i = (size_t)row * 9 + lane;
        v[0] += A.r[i] * A.h[i];
      }
    if (!exchange_sum<3, P64_W>(bar, A.red2, v, X2)) {
      drain();
      return;
    }
    if (threadIdx.x == 0) {
      sc[0][0] = sc[0][1] = v[0];
      sc[0][2] = sc[0][3] = 1.e50;
    }
  }
  if (RES && T > 0) {
    ok = stage_wait(A, mbar, 0u);
    landed = true;
  }
  double beta_prev = 0.;
  bool converged = false;
  int k;
  for (k = 0; k < A.msize; ++k) {
    const double *dprev = (k & 1) ? A.D0 : A.D1;
    double *dcur = (k & 1) ? A.D1 : A.D0;
    // ---- phase 1
    double pdq[1] = {0.};
    if constexpr (SYM) {
      // 1a: both products of every block; the even warp of a stage B d_col,
      // the odd one B^T d_row
      if (stream) {
        const int tr = warp & 1;
        double *buf = (double *)(stg + P1S_BLK + P1S_IDX + tr * 2 * P1S_BUF), *bufd = buf + 32 * 9;
        const int4 *idx = (const int4 *)(stg + P1S_BLK);
        for (int g = gs; g < ng; g += gstep) {
          const Grp64 q = group64(A, g);
          if (ok && (!keep || k == 0)) ok = stage_wait(A, mbar, parity);
          const unsigned mis = (unsigned)(((unsigned long long)A.blocks + (unsigned long long)q.start * 648u) & 15ull);
          if (ok && !(tr && q.diag)) {
            // the 32 vectors d^k = h + beta d^(k-1): all the copies of both
            // parts in flight, three vectors an instruction
#pragma unroll
            for (int m = 0; m < 11; ++m) {
              const int v = 3 * m + grp;
              if (lane < 27 && v < q.n) {
                const size_t o = (size_t)(tr ? idx[v].x : idx[v].y) * 9 + rr;
                cp_async8(buf + v * 9 + rr, A.h + o);
                cp_async8(bufd + v * 9 + rr, dprev + o);
              }
            }
            cp_async_wait_all();
            __syncwarp();
            const double *B = (const double *)(stg + mis + 648 * lane);
            double dv[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) dv[j] = buf[lane * 9 + j] + beta_prev * bufd[lane * 9 + j];
            if (q.diag && lane < q.n)  // d^k of every row
#pragma unroll
              for (int j = 0; j < 9; ++j) dcur[(size_t)idx[lane].x * 9 + j] = dv[j];
            __syncwarp();
            if (lane < q.n) {
              if (!tr) {
#pragma unroll 3
                for (int i = 0; i < 9; ++i) {
                  double acc = 0.;
#pragma unroll
                  for (int j = 0; j < 9; ++j) acc += B[i * 9 + j] * dv[j];
                  buf[lane * 9 + i] = acc;
                }
              } else {
#pragma unroll 3
                for (int j = 0; j < 9; ++j) {
                  double acc = 0.;
#pragma unroll
                  for (int i = 0; i < 9; ++i) acc += B[i * 9 + j] * dv[i];
                  buf[lane * 9 + j] = acc;
                }
              }
            }
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 11; ++m) {
              const int v = 3 * m + grp;
              if (lane < 27 && v < q.n) A.prod[(size_t)(tr ? idx[v].w : idx[v].z) * 9 + rr] = buf[v * 9 + rr];
            }
          }
          if (!keep) {
            // both warps are done with the stage: the next group, or the
            // first one for the next iteration
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
            parity ^= 1u;
            if (ok && lane == 0 && !tr) {
              fence_proxy_async();
              group64_issue(A, g + gstep < ng ? g + gstep : gs, stg, mbar, policy);
            }
          }
          __syncwarp();
        }
      }
      // the items' records of 1b (constant) ahead of the barrier
      int2 m[4];
      auto load_recs = [&](int t) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          m[j] = t + j < T ? __ldg(A.item_rec + (size_t)gwarp + (size_t)(t + j) * nwarps) : make_int2(0, 0);
      };
      load_recs(0);
      if (!ok && lane == 0) atomicOr(A.err, 2);
      if (!bar.sync(!ok)) {
        drain();
        return;
      }
      // 1b: the items' sums, four items' loads in flight beside the next
      // four's records
      for (int t = 0; t < T; t += 4) {
        double u[4], dk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          u[j] = lane < 27 && grp < (m[j].x >> 16) ? __ldcg(A.prod + (size_t)(m[j].y + grp) * 9 + rr) : 0.;
          dk[j] = lane < 9 && t + j < T ? __ldcg(dcur + (size_t)(m[j].x & 0xffff) * 9 + lane) : 0.;
        }
        if (t + 4 < T) load_recs(t + 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double a1 = __shfl_down_sync(0xffffffffu, u[j], 9);
          const double a2 = __shfl_down_sync(0xffffffffu, u[j], 18);
          if (lane < 9 && t + j < T) {
            const double p = u[j] + a1 + a2;
            A.part[((size_t)gwarp + (size_t)(t + j) * nwarps) * 9 + lane] = p;
            pdq[0] += dk[j] * p;
          }
        }
      }
    } else if constexpr (RES) {
      double hc[P1_SLOTS], dc[P1_SLOTS], hk[P1_SLOTS], dk[P1_SLOTS];
#pragma unroll
      for (int t = 0; t < P1_SLOTS; ++t) {
        hc[t] = dc[t] = hk[t] = dk[t] = 0.;
        if (t < T) {
          const int meta = recs[4 * t].x;
          if (lane < 27 && grp < (meta >> 16)) {
            const size_t j = (size_t)recs[4 * t + 1 + grp].x * 9 + rr;
            hc[t] = __ldcg(A.h + j);
            dc[t] = __ldcg(dprev + j);
          }
          if (lane < 9) {
            const size_t i = (size_t)(meta & 0xffff) * 9 + lane;
            hk[t] = __ldcg(A.h + i);
            dk[t] = __ldcg(dprev + i);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < P1_SLOTS; ++t)
        if (t < T) {
          const int en = recs[4 * t + 1 + (grp < 3 ? grp : 0)].y;
          const bool act = lane < 27 && grp < (recs[4 * t].x >> 16);
          const bool tr = en < 0;
          const double *B = (const double *)(stg + (3 * t + (grp < 3 ? grp : 0)) * P1_PIECE + ((en & 1) << 3));
          const double cdc = hc[t] + beta_prev * dc[t];
          double acc = 0.;
#pragma unroll
          for (int c = 0; c < 9; ++c) {
            const double xc = __shfl_sync(0xffffffffu, cdc, (lane < 27 ? gbase : 0) + c);
            if (act) acc += B[tr ? c * 9 + rr : rr * 9 + c] * xc;
          }
          const double a1 = __shfl_down_sync(0xffffffffu, acc, 9);
          const double a2 = __shfl_down_sync(0xffffffffu, acc, 18);
          if (lane < 9) {
            const double p = acc + a1 + a2;
            A.part[((size_t)gwarp + (size_t)t * nwarps) * 9 + lane] = p;
            const double dkv = hk[t] + beta_prev * dk[t];
            pdq[0] += dkv * p;
          }
        }
      if (!ok && lane == 0) atomicOr(A.err, 2);
    } else {
      const int gl = grp < 3 ? grp : 0;
      for (int t = 0; t < T; ++t) {
        const size_t item = (size_t)gwarp + (size_t)t * nwarps;
        const int2 m = __ldg(A.item_rec + item);
        const bool act = lane < 27 && grp < (m.x >> 16);
        const int2 en = act ? __ldg(A.ent + m.y + grp) : make_int2(0, 0);
        const bool tr = en.y < 0;
        const double *B = (const double *)A.blocks + (size_t)(en.y & 0x7fffffff) * 81;
        double bv[9], cdc = 0.;
#pragma unroll
        for (int c = 0; c < 9; ++c) bv[c] = act ? __ldg(B + (tr ? c * 9 + rr : rr * 9 + c)) : 0.;
        if (act) {
          const size_t j = (size_t)en.x * 9 + rr;
          cdc = __ldcg(A.h + j) + beta_prev * __ldcg(dprev + j);
        }
        double acc = 0.;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const double xc = __shfl_sync(0xffffffffu, cdc, 9 * gl + c);
          if (act) acc += bv[c] * xc;
        }
        const double a1 = __shfl_down_sync(0xffffffffu, acc, 9);
        const double a2 = __shfl_down_sync(0xffffffffu, acc, 18);
        if (lane < 9) {
          const size_t i = (size_t)(m.x & 0xffff) * 9 + lane;
          const double p = acc + a1 + a2;
          A.part[item * 9 + lane] = p;
          const double dkv = __ldcg(A.h + i) + beta_prev * __ldcg(dprev + i);
          pdq[0] += dkv * p;
        }
      }
    }
    // this warp's vectors of its first row, ahead of the exchange
    // (streamed form: d^k itself, stored in phase 1a)
    double hva = 0., dpa = 0., xva = 0., rva = 0.;
    if (has_row && lane < 9) {
      const size_t i = (size_t)rowa * 9 + lane;
      hva = __ldcg(A.h + i);
      dpa = __ldcg((SYM ? dcur : dprev) + i);
      xva = A.x[i];
      rva = A.r[i];
    }
    if (!exchange_sum<1, P64_W>(bar, A.red1, pdq, X1, !ok)) {
      drain();
      return;
    }
    const double edtAdk = pdq[0], erthk = sc[k & 1][0];
    double alpha;
    if (fabs(erthk) < 1.e-20 || fabs(erthk) > 1.e20)
      alpha = 0.;
    else
      alpha = erthk / edtAdk;
    // ---- phase 2
    double p2[3] = {0., 0., 0.};
    if constexpr (!CO) {
      for (int row = rowa; row < A.row1; row += nwarps) {
        const bool first = row == rowa;
        const size_t i = (size_t)row * 9 + (lane < 9 ? lane : 0);
        double r1v = 0., hv = 0.;
        const int t0 = first ? ta0 : A.row_item_off[row], t1 = first ? ta1 : A.row_item_off[row + 1];
        const double q = row_q(A, t0, t1, lane, grp, rr);
        if (lane < 9) {
          hv = first ? hva : __ldcg(A.h + i);
          double dk;
          if constexpr (SYM) {
            dk = first ? dpa : __ldcg(dcur + i);
          } else {
            dk = hv + beta_prev * (first ? dpa : __ldcg(dprev + i));
            dcur[i] = dk;
          }
          A.x[i] = (first ? xva : A.x[i]) + alpha * dk;
          const double dr = alpha * q;
          r1v = (first ? rva : A.r[i]) - dr;
          p2[0] += dr * dr;
        }
        const double *C = RES && first ? Cs : A.Cinv + (size_t)row * 81;
        double h1v = 0.;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const double rc = __shfl_sync(0xffffffffu, r1v, c);
          if (lane < 9) h1v += C[lane * 9 + c] * rc;
        }
        if (lane < 9) {
          A.r[i] = r1v;
          A.h[i] = h1v;
          p2[1] += r1v * (h1v - hv);
          p2[2] += r1v * h1v;
        }
      }
    } else {
      __shared__ double shr[P64_W][CO_M];
      __shared__ double shz[CO_M];
      for (int a = blockIdx.x; a < A.nagg; a += G) {
        const int t0 = A.agg_off[a], t1 = A.agg_off[a + 1];
        double rcw = 0.;
        for (int t = t0 + warp; t < t1; t += P64_W) {
          const int row = A.agg_rows[t];
          const size_t i = (size_t)row * 9 + (lane < 9 ? lane : 0);
          double r1v = 0.;
          const double q = row_q(A, A.row_item_off[row], A.row_item_off[row + 1], lane, grp, rr);
          if (lane < 9) {
            double dk;
            if constexpr (SYM) {
              dk = __ldcg(dcur + i);
            } else {
              dk = __ldcg(A.h + i) + beta_prev * __ldcg(dprev + i);
              dcur[i] = dk;
            }
            A.x[i] = __ldcg(A.x + i) + alpha * dk;
            const double dr = alpha * q;
            r1v = __ldcg(A.r + i) - dr;
            p2[0] += dr * dr;
          }
          const double *C = A.Cinv + (size_t)row * 81;
          const double *Pk = A.P + (size_t)row * (9 * CO_M);
          double h1v = 0.;
#pragma unroll
          for (int c = 0; c < 9; ++c) {
            const double rc = __shfl_sync(0xffffffffu, r1v, c);
            if (lane < 9) h1v += __ldg(C + lane * 9 + c) * rc;
            if (lane < CO_M) rcw += __ldg(Pk + c * CO_M + lane) * rc;
          }
          if (lane < 9) {
            A.r[i] = r1v;
            A.hj[i] = h1v;
          }
        }
        if (lane < CO_M) shr[warp][lane] = rcw;
        __syncthreads();
        if (threadIdx.x < CO_M) {
          double sum = 0.;
          for (int w = 0; w < P64_W; ++w) sum += shr[w][threadIdx.x];
          A.rc[a * CO_M + threadIdx.x] = sum;
        }
        __syncthreads();
      }
      if (!bar.sync()) {
        drain();
        return;
      }
      for (int a = blockIdx.x; a < A.nagg; a += G) {
        double z[CO_M];
#pragma unroll
        for (int j = 0; j < CO_M; ++j) z[j] = 0.;
        for (int i = threadIdx.x; i < A.nc; i += P64_T) {
          const double rv = __ldcg(A.rc + i);
#pragma unroll
          for (int j = 0; j < CO_M; ++j) z[j] += __ldg(A.Ainv + (size_t)(a * CO_M + j) * A.nc + i) * rv;
        }
#pragma unroll
        for (int j = 0; j < CO_M; ++j) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) z[j] += __shfl_xor_sync(0xffffffffu, z[j], o);
          if (lane == 0) shr[warp][j] = z[j];
        }
        __syncthreads();
        if (threadIdx.x < CO_M) {
          double sum = 0.;
          for (int w = 0; w < P64_W; ++w) sum += shr[w][threadIdx.x];
          shz[threadIdx.x] = sum;
        }
        __syncthreads();
        const int t0 = A.agg_off[a], t1 = A.agg_off[a + 1];
        for (int t = t0 + warp; t < t1; t += P64_W) {
          const int row = A.agg_rows[t];
          if (lane < 9) {
            const size_t i = (size_t)row * 9 + lane;
            const double *Pk = A.P + (size_t)row * (9 * CO_M) + lane * CO_M;
            double h1v = __ldcg(A.hj + i);
#pragma unroll
            for (int j = 0; j < CO_M; ++j) h1v += __ldg(Pk + j) * shz[j];
            const double hv = __ldcg(A.h + i), r1v = __ldcg(A.r + i);
            p2[1] += r1v * (h1v - hv);
            p2[2] += r1v * h1v;
            A.h[i] = h1v;
          }
        }
        __syncthreads();
      }
    }
    if (!exchange_sum<3, P64_W>(bar, A.red2, p2, X2)) {
      drain();
      return;
    }
    const double(&g3)[3] = p2;
    const double meandr = g3[0], er1th1 = g3[1];
    const double erthk0 = sc[k & 1][1], meandrold = sc[k & 1][2], meandr0 = k == 0 ? meandr : sc[k & 1][3];
    // mode 0 keeps the iterate with the smallest increment (the reference's
    // exivold); mode 1 keeps the latest finite one and stops, unconverged,
    // at a breakdown (a non-finite residual or increment)
    const bool finite = isfinite(g3[0]) && isfinite(g3[2]);
    const bool improved = (A.mode == 1 && finite) || meandr < meandrold;
    if (improved) {
      for (int row = A.row0 + gwarp; row < A.row1; row += nwarps)
        if (lane < 9) A.xbest[(size_t)row * 9 + lane] = __ldcg(A.x + (size_t)row * 9 + lane);
    }
    if (A.mode == 0 && meandr * 1.e5 < meandr0) break;
    if (A.mode == 1 && !finite) break;
    if (A.mode == 1 && g3[2] <= A.tol2 * erthk0) {
      converged = true;
      break;
    }
    double beta = fabs(er1th1) < 1.e-10 ? 0. : er1th1 / sc[k & 1][0];
    if (beta < 0.) beta = 0.;
    beta_prev = beta;
    if (threadIdx.x == 0) {
      sc[(k + 1) & 1][0] = g3[2];
      sc[(k + 1) & 1][1] = erthk0;
      sc[(k + 1) & 1][2] = improved ? meandr : meandrold;
      sc[(k + 1) & 1][3] = meandr0;
    }
  }
  drain();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.iters[0] = k < A.msize ? k + 1 : A.msize;
    A.iters[1] = converged ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------
// The FP32 form's persistent PCG (mixed precision and the learned solver).
//
// Phase 1 streams the reduced camera system through shared memory with 1-D
// TMA bulk copies.  The blocks are read in storage order: the diagonal
// blocks of rows begini.. first, then every off-diagonal block once (upper
// triangle, row major).  The stream is cut into groups of 32 blocks and the
// groups into chunks of A.chunk groups (fixed boundaries); warps take chunks
// from a counter, the next one taken a chunk ahead, so a fast warp takes
// more of them.  One elected lane copies a group's blocks (32 x 324 B) and
// their (row, column, slot) triples into the warp's stage, completing on the
// stage's mbarrier; each lane then owns one block: it forms the block's row
// product B d_col (summed into its row) and, for an off-diagonal block, the
// transposed product B^T d_row, which goes to the block's slot of tpart.
// The slots are in column order (the blocks of column c, i.e. the
// transposed entries of row c, are consecutive), and a slot is 64 bytes (9
// values, zero padding: two whole sectors, so the scattered writes need no
// read of the rest of a sector), so that phase 2 reads each row's
// transposed products as one contiguous run.  Lane i reads its block at byte
// 324 i of the stage: 81 i is a distinct bank for every lane, so the reads
// are conflict-free.  The gathered vector is d^k rounded to FP32 (d32, 12
// floats per camera so that a camera is three aligned 16-byte loads),
// formed for all rows in phase D before phase 1.
//
// Row sums: a diagonal block's product is written to pdiag[row]; the
// off-diagonal products of a row are summed per group by a segmented warp
// scan in FP32 (a group inside the open row: per-lane FP64 running sums),
// carried across groups in FP64 and written once per (row, chunk): to
// prow[row] by the chunk that holds the row's first block, to pw[chunk] by a
// chunk that starts inside the row; each chunk's share of d^T A d goes to
// pdqc[chunk].  Everything a chunk writes depends on the chunk only, not on
// the warp that took it.  Phase 2 adds, per row and in a fixed order, pdiag,
// prow, the pw of the chunks that start inside the row, and the row's run of
// transposed products (the blocks stored by earlier rows in its column).
//
// Iteration k: phase D (d^k = h + beta d^(k-1), FP64 and FP32 copies),
// barrier, phase 1 (A d^k and d^T A d), barrier, phase 2 (as in the FP64
// form; with the coarse space: 2a, rows taken from a counter, barrier, 2a',
// the aggregates' restrictions, barrier, 2b, the coarse correction),
// barrier.
constexpr int P32_W = 16;  // warps per CTA
constexpr int P32_T = P32_W * 32;
constexpr int GB = 32;     // blocks per group: one per lane
constexpr int STG_BLK = GB * 324 + 16;
constexpr int STG_IDX = GB * 16;
constexpr int STG_BYTES = STG_BLK + STG_IDX + 16;  // + the mbarrier
constexpr size_t P32_SMEM = (size_t)P32_W * STG_BYTES;
static_assert(STG_BLK % 16 == 0 && STG_IDX % 16 == 0, "16-byte aligned stage parts");

// Group g of the stream: its first block (storage index), its block count
// and, for an off-diagonal group, the first block's off-diagonal index.
struct Grp32 {
  long long start;
  int n;
  bool diag;
  long long boff;
};
__device__ __forceinline__ Grp32 group_of(long long g, int gd, int row0, int row1, int nboff) {
  Grp32 q;
  if (g < gd) {
    q.start = row0 + GB * g;
    q.n = (int)min((long long)GB, row1 - q.start);
    q.diag = true;
    q.boff = -1;
  } else {
    const long long j = g - gd;
    q.boff = GB * j;
    q.start = row1 + q.boff;
    q.n = (int)min((long long)GB, nboff - q.boff);
    q.diag = false;
  }
  return q;
}
// Phase 1 is cut into chunks of A.chunk groups (fixed boundaries); the warps take
// chunks from a counter, so a fast warp takes more of them, and everything a
// chunk writes (its row sums, its share of d^T A d) depends only on the
// chunk: the result does not depend on which warp took it.

// Byte offsets of a group's data inside its 16-byte aligned copies.
__device__ __forceinline__ unsigned blk_misalign(const float *blocks, long long start) {
  return (unsigned)(((unsigned long long)(blocks + start * 81)) & 15ull);
}
constexpr int TP_STRIDE = 16;  // floats per transposed-product slot (64 B)
constexpr int RC_S = 12;       // doubles per row of rowc

// Issue the copies of group q into the warp's stage (one lane).
__device__ __forceinline__ void group_issue(const PcgArgs &A, const Grp32 &q, unsigned char *stg,
                                            unsigned long long *bar) {
  const float *blocks = (const float *)A.blocks;
  const unsigned mb = blk_misalign(blocks, q.start);
  const unsigned nb_bytes = (mb + (unsigned)q.n * 324u + 15u) & ~15u;
  const unsigned ni_bytes = (unsigned)q.n * 16u;
  mbar_expect_tx(bar, nb_bytes + ni_bytes + tx_extra(A));
  bulk_load(stg, (const unsigned char *)(blocks + q.start * 81) - mb, nb_bytes, bar);
  bulk_load(stg + STG_BLK, A.bidx + q.start, ni_bytes, bar);
}

// FP32 d^k of camera c (12-float stride) into v[0..8].  The loads may hit
// L1: d32 is written in phase D by all CTAs before a grid barrier, whose
// release arrivals, acquiring load (thread 0's) and block barrier order those
// writes before these loads, and the rows of a cluster keep gathering the
// same columns.
__device__ __forceinline__ void load_d32(const float *d32, int c, float (&v)[9]) {
  const float4 *p = (const float4 *)(d32 + (size_t)c * 12);
  const float4 a = __ldca(p), b = __ldca(p + 1), e = __ldca(p + 2);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  v[8] = e.x;
}

// The butterfly sums (lanes xor 16, 8, 4, 2, 1) of M <= 16 values over the
// warp: value j ends in lanes 2 j and 2 j + 1.  Each step passes on the half
// of the values its partner keeps, 16 exchanges instead of 5 M; every value
// is added in the order of the full butterfly (a + b = b + a), so the result
// is the same to the bit.
template <int M>
__device__ __forceinline__ double butterfly_scatter(const double (&v)[M], int lane) {
  double w[8];
  {
    const bool up = lane & 16;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double lo = j < M ? v[j < M ? j : 0] : 0., hi = j + 8 < M ? v[j + 8 < M ? j + 8 : 0] : 0.;
      w[j] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, 16);
    }
  }
#pragma unroll
  for (int o = 8, n = 4; o > 1; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < n) w[j] = (up ? w[j + n] : w[j]) + __shfl_xor_sync(0xffffffffu, up ? w[j] : w[j + n], o);
  }
  return w[0] + __shfl_xor_sync(0xffffffffu, w[0], 1);
}

// q of one row in lanes < 9 (FP32 form).
__device__ __forceinline__ double row_q32(const PcgArgs &A, int row, long long gd, long long ch, int lane) {
  // the row's run of transposed products (slots firstT[row] ..
  // firstT[row + 1]): one slot per lane (three 16-byte loads), and the sums
  // of the phase-1 chunks that start strictly inside the row's off-diagonal
  // blocks, one chunk per lane; nine FP64 partial sums, then a fixed butterfly
  double acc[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) acc[j] = 0.;
  const int e0 = __ldg(A.firstT + row), e1 = __ldg(A.firstT + row + 1);
  const int f0 = __ldg(A.firstN + row), f1 = __ldg(A.firstN + row + 1);
#pragma unroll 4
  for (int e = e0 + lane; e < e1; e += 32) {
    const float4 *t = (const float4 *)(A.tpart + (size_t)e * TP_STRIDE);
    const float4 a = __ldcg(t), b = __ldcg(t + 1), c = __ldcg(t + 2);
    acc[0] += (double)a.x;
    acc[1] += (double)a.y;
    acc[2] += (double)a.z;
    acc[3] += (double)a.w;
    acc[4] += (double)b.x;
    acc[5] += (double)b.y;
    acc[6] += (double)b.z;
    acc[7] += (double)b.w;
    acc[8] += (double)c.x;
  }
  if (f1 > f0) {
    const long long glo = gd + f0 / GB + 1, ghi = gd + (f1 - 1) / GB;
    for (long long c = (glo + ch - 1) / ch + lane; c * ch <= ghi; c += 32) {
      const double *w = A.pw + (size_t)c * 9;
#pragma unroll
      for (int j = 0; j < 9; ++j) acc[j] += __ldcg(w + j);
    }
  }
  double q = __shfl_sync(0xffffffffu, butterfly_scatter<9>(acc, lane), 2 * (lane < 9 ? lane : 0));
  if (lane < 9) {
    const size_t i = (size_t)row * 9 + lane;
    q += __ldcg(A.pdiag + i);
    if (f1 > f0) q += __ldcg(A.prow + i);
  }
  return q;
}

// Both products of the lane's block of the group in the stage: y = B d_col
// and, off the diagonal, t = B^T d_row; pdq += d_row^T y (+ d_col^T t).
__device__ __forceinline__ void group_products(const PcgArgs &A, const Grp32 &q, const unsigned char *stg, int lane,
                                               bool act, int4 &rc, float (&y)[9], float (&t)[9], double &pdq) {
  const unsigned mb = blk_misalign((const float *)A.blocks, q.start);
  float dc[9], dr[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    y[j] = 0.f;
    t[j] = 0.f;
  }
  if (act) {
    rc = *(const int4 *)(stg + STG_BLK + 16 * lane);
    load_d32(A.d32, rc.y, dc);
    load_d32(A.d32, rc.x, dr);
    const float *B = (const float *)(stg + mb + 324 * lane);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      float yi = 0.f;
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const float b = B[i * 9 + j];
        yi = fmaf(b, dc[j], yi);
        t[j] = fmaf(b, dr[i], t[j]);
      }
      y[i] = yi;
    }
    double s = 0.;
#pragma unroll
    for (int i = 0; i < 9; ++i) s += (double)dr[i] * (double)y[i];
    if (!q.diag)
#pragma unroll
      for (int j = 0; j < 9; ++j) s += (double)dc[j] * (double)t[j];
    pdq += s;
  }
}
// The transposed product to its slot (column order).
__device__ __forceinline__ void store_transposed(const PcgArgs &A, int slot, const float (&t)[9]) {
  float4 *dst = (float4 *)(A.tpart + (size_t)slot * TP_STRIDE);
  __stcg(dst, make_float4(t[0], t[1], t[2], t[3]));
  __stcg(dst + 1, make_float4(t[4], t[5], t[6], t[7]));
  __stcg(dst + 2, make_float4(t[8], 0.f, 0.f, 0.f));
  __stcg(dst + 3, make_float4(0.f, 0.f, 0.f, 0.f));
}
// Inclusive scan of y over the lanes of equal row (rows non-decreasing in
// lane order; inactive lanes carry distinct negative rows).
__device__ __forceinline__ void segment_scan(int row, float (&y)[9], int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ru = __shfl_up_sync(0xffffffffu, row, o);
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const float vu = __shfl_up_sync(0xffffffffu, y[j], o);
      if (lane >= o && ru == row) y[j] += vu;
    }
  }
}

// SMALL: systems of at most one group per warp.  Four warps (a quad) take a
// chunk, a group each, which stays in the warp's stage for the whole solve;
// the quads are dealt over the CTAs.  Sums that lie inside a group are
// written by the lane that ends them; a row's run across the quad's groups is
// put together by the quad's first warp from its pieces in shared memory, in
// the order and precision of the one-warp form (a group inside the row in
// FP64 per lane, the others by the FP32 scan), so that both forms give the
// same bits.  With the coarse space an aggregate's CTA takes its rows itself
// and sums their restrictions (2a and 2a' in one).  Such a system is latency:
// with a chunk's groups one after the other in a warp, on as few CTAs as hold
// the chunks, 3,000 cameras (944 groups) took 117,000 cycles an iteration,
// 44,000 of them in phase 1; now 42,000 (57.0 -> 20.7 ms a solve).
struct Quad {
  float y[4][32 * 9];  // a group inside a row: every lane's product; else the first and last segments' sums
  double s[4][32];     // the lanes' shares of d^T A d
  int flags[4], row[4];
};
constexpr int QF_OFF = 1, QF_INSIDE = 2, QF_NEXT = 4, QF_HEAD = 8;
template <bool CO, bool SMALL>
__global__ void __launch_bounds__(P32_T, 1) k_pcg32(PcgArgs A) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gwarp = blockIdx.x * P32_W + warp, nwarps = gridDim.x * P32_W;
  const int G = gridDim.x;
  GridBarrier bar(A.bar, (unsigned)G + A.bar_extra, A.err, A.bar_ns);
  __shared__ Exchange<3, P32_W> X2;
  __shared__ double sh[P32_W + 1];
  extern __shared__ __align__(16) unsigned char pcg_dyn[];
  unsigned char *stg = pcg_dyn + (size_t)warp * STG_BYTES;
  unsigned long long *mbar = (unsigned long long *)(stg + STG_BLK + STG_IDX);
  unsigned parity = 0;
  if (lane == 0) mbar_init(mbar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  __syncwarp();
  const long long gd = (A.row1 - A.row0 + GB - 1) / GB, go = ((long long)A.nboff + GB - 1) / GB;
  const long long ng = gd + go, ch = A.chunk, nch = (ng + ch - 1) / ch;
  // rows whose contributions to the sums a warp adds (the sums' order): with
  // SMALL the first g0 CTAs, those the one-warp form would take
  const int nrw = SMALL ? (int)A.g0 * P32_W : nwarps, row_a = SMALL && gwarp >= nrw ? A.row1 : A.row0 + gwarp;
  // SMALL: the quad's chunk and the warp's group of it
  __shared__ Quad quads[SMALL ? P32_W / 4 : 1];
  Quad &Q = quads[SMALL ? warp >> 2 : 0];
  const int qp = warp & 3, qc = (warp >> 2) * G + (int)blockIdx.x;
  const bool has_group = SMALL && qc < nch && 4ll * qc + qp < ng;
  int qrow_prev = -1, qrow_next = -1;  // the rows next to the group in its chunk
  if constexpr (SMALL) {
    if (lane == 0) Q.flags[qp] = 0;
    Q.s[qp][lane] = 0.;
    if (has_group) {
      const long long g = 4ll * qc + qp;
      const Grp32 q = group_of(g, (int)gd, A.row0, A.row1, A.nboff);
      if (lane == 0) group_issue(A, q, stg, mbar);
      if (!q.diag) {
        const int r0 = A.bidx[q.start].x, r1 = A.bidx[q.start + q.n - 1].x;
        if (qp > 0 && g - 1 >= gd) qrow_prev = A.bidx[q.start - 1].x;
        if (qp < 3 && g + 1 < ng) qrow_next = A.bidx[q.start + q.n].x;
        if (lane == 0) {
          Q.row[qp] = r1;
          Q.flags[qp] = QF_OFF | (r0 == r1 && r0 == qrow_prev ? QF_INSIDE : 0) | (r1 == qrow_next ? QF_NEXT : 0) |
                        (r0 != r1 || qrow_prev >= 0 || q.boff == (long long)A.firstN[r1] ? QF_HEAD : 0);
        }
      }
    }
  }
  // r^T h of the start vectors
  double erthk;
  {
    double v[3] = {0., 0., 0.};
    for (int row = row_a; row < A.row1; row += nrw)
      if (lane < 9) {
        const size_t i = (size_t)row * 9 + lane;
        v[0] += A.r[i] * A.h[i];
      }
    // (the group's copy ends before the kernel can)
    const bool landed = !has_group || stage_wait(A, mbar, 0u);
    if (!landed) {
      if (lane == 0) atomicOr(A.err, 2);
      stage_wait(A, mbar, 0u);
    }
    if (!exchange_sum<3, P32_W>(bar, A.red2, v, X2, !landed)) return;
    erthk = v[0];
  }
  double meandrold = 1.e50, meandr0 = 1.e50, beta_prev = 0.;
  const double erthk0 = erthk;
  bool converged = false;
  int k;
  for (k = 0; k < A.msize; ++k) {
    const double *dprev = (k & 1) ? A.D0 : A.D1;
    double *dcur = (k & 1) ? A.D1 : A.D0;
    // ---- phase D: d^k for every row, FP64 and FP32
    for (int row = A.row0 + (SMALL ? warp * G + (int)blockIdx.x : gwarp); row < A.row1; row += nwarps)
      if (lane < 9) {
        const size_t i = (size_t)row * 9 + lane;
        const double dk = __ldcg(A.h + i) + beta_prev * __ldcg(dprev + i);
        dcur[i] = dk;
        A.d32[(size_t)row * 12 + lane] = (float)dk;
      }
    if (!SMALL && blockIdx.x == 0 && threadIdx.x < 2) A.ctr[threadIdx.x] = 0u;
    if (!bar.sync()) return;
    // ---- phase 1
    bool ok = true;
    if constexpr (SMALL) {
      if (has_group) {
        const Grp32 q = group_of(4ll * qc + qp, (int)gd, A.row0, A.row1, A.nboff);
        const bool act = lane < q.n;
        int4 rc = make_int4(-1 - lane, -1, 0, 0);
        float y[9], t[9];
        double pdq = 0.;
        group_products(A, q, stg, lane, act, rc, y, t, pdq);
        Q.s[qp][lane] = pdq;
        if (q.diag) {
          if (act) {
            double *dst = A.pdiag + (size_t)rc.x * 9;
#pragma unroll
            for (int i = 0; i < 9; ++i) dst[i] = (double)y[i];
          }
        } else {
          if (act) store_transposed(A, rc.z, t);
          if (Q.flags[qp] & QF_INSIDE) {
#pragma unroll
            for (int j = 0; j < 9; ++j) Q.y[qp][lane * 9 + j] = act ? y[j] : 0.f;
          } else {
            const int row = rc.x;
            segment_scan(row, y, lane);
            const int rnext = __shfl_down_sync(0xffffffffu, row, 1), r0 = __shfl_sync(0xffffffffu, row, 0);
            const bool last = lane == q.n - 1;
            if (act && (last || rnext != row)) {
              const bool first = row == r0;
              const bool piece_p = first && row == qrow_prev, piece_n = last && row == qrow_next;
              if (piece_p || piece_n) {
                // (both only if the group lies inside the row)
                float *dst = Q.y[qp] + (piece_n ? 16 : 0);
#pragma unroll
                for (int j = 0; j < 9; ++j) dst[j] = y[j];
              } else {
                // a segment starts the row unless it is the chunk's first and
                // the row began before the chunk
                const bool head = !first || qrow_prev >= 0 || q.boff == (long long)__ldg(A.firstN + row);
                double *dst = head ? A.prow + (size_t)row * 9 : A.pw + (size_t)qc * 9;
#pragma unroll
                for (int j = 0; j < 9; ++j) dst[j] = (double)y[j];
              }
            }
          }
        }
      }
      if (qc < nch) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp >> 2)) : "memory");
        if (qp == 0) {
          // rows that run on from one group of the chunk to the next
          bool open = false, head = false;
          int row = -1;
          double racc = 0.;
#pragma unroll 1
          for (int p = 0; p < 4; ++p) {
            const int f = Q.flags[p];
            if (!(f & QF_OFF)) continue;
            if (open) {
              if (f & QF_INSIDE) {
                // the lanes' sums over the groups inside the row, folded at its end
                double l[9];
#pragma unroll
                for (int j = 0; j < 9; ++j) l[j] = 0.;
                for (; p < 4 && (Q.flags[p] & QF_INSIDE); ++p) {
#pragma unroll
                  for (int j = 0; j < 9; ++j) l[j] += (double)Q.y[p][lane * 9 + j];
                  if (!(Q.flags[p] & QF_NEXT)) {
                    open = false;
                    break;
                  }
                }
                racc += __shfl_sync(0xffffffffu, butterfly_scatter<9>(l, lane), 2 * (lane < 9 ? lane : 0));
                if (open && p < 4) racc += lane < 9 ? (double)Q.y[p][lane] : 0.;  // its last, partial group
              } else {
                racc += lane < 9 ? (double)Q.y[p][lane] : 0.;
              }
              open = false;
              if (lane < 9) (head ? A.prow + (size_t)row * 9 : A.pw + (size_t)qc * 9)[lane] = racc;
              if (p >= 4) break;
            }
            const int g = Q.flags[p];
            if ((g & QF_NEXT) && !(g & QF_INSIDE)) {
              open = true;
              head = g & QF_HEAD;
              row = Q.row[p];
              racc = lane < 9 ? (double)Q.y[p][16 + lane] : 0.;
            }
          }
          double pdq = 0.;
#pragma unroll
          for (int p = 0; p < 4; ++p) pdq += Q.s[p][lane];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) pdq += __shfl_xor_sync(0xffffffffu, pdq, o);
          if (lane == 0) A.pdqc[qc] = pdq;
        }
      }
    } else {
      auto grab = [&]() -> long long {
        unsigned c = 0;
        if (lane == 0) c = atomicAdd(A.ctr, 1u);
        return (long long)__shfl_sync(0xffffffffu, c, 0);
      };
      long long c = grab();
      long long cn = c < nch ? grab() : nch;  // the next chunk, taken one ahead
      int cur_row = -1;   // row of the running sum (-1: none yet in this chunk)
      bool cur_head = false;
      double racc = 0.;   // running sum of cur_row, component `lane` (lanes < 9)
      double pdq = 0.;    // this chunk's share of d^T A d (per lane)
      auto flush = [&]() {
        if (cur_row >= 0 && lane < 9) {
          double *dst = cur_head ? A.prow + (size_t)cur_row * 9 : A.pw + (size_t)c * 9;
          dst[lane] = racc;
        }
      };
      // per-lane running sums of the open row over the groups inside it,
      // folded into racc (lanes 0..8) at the row's end in a fixed butterfly
      double lacc[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) lacc[j] = 0.;
      auto fold_lanes = [&]() {
        const double v = butterfly_scatter<9>(lacc, lane);
#pragma unroll
        for (int j = 0; j < 9; ++j) lacc[j] = 0.;
        const double vl = __shfl_sync(0xffffffffu, v, 2 * (lane < 9 ? lane : 0));
        racc += lane < 9 ? vl : 0.;
      };
      if (c < nch && lane == 0) group_issue(A, group_of(c * ch, (int)gd, A.row0, A.row1, A.nboff), stg, mbar);
      while (c < nch) {
        const long long g0 = c * ch, g1 = min(ng, g0 + ch);
        cur_row = -1;
        racc = 0.;
        pdq = 0.;
        for (long long g = g0; g < g1; ++g) {
          const Grp32 q = group_of(g, (int)gd, A.row0, A.row1, A.nboff);
          if (!stage_wait(A, mbar, parity)) {
            ok = false;
            break;
          }
          parity ^= 1u;
          const bool act = lane < q.n;
          int4 rc = make_int4(-1 - lane, -1, 0, 0);
          float y[9], t[9];
          group_products(A, q, stg, lane, act, rc, y, t, pdq);
          // the stage's blocks are read: the next group's copies may land
          // (the next group of this chunk, or the first of the next chunk)
          __syncwarp();
          const long long gn = g + 1 < g1 ? g + 1 : (cn < nch ? cn * ch : -1);
          if (lane == 0 && gn >= 0) {
            fence_proxy_async();
            group_issue(A, group_of(gn, (int)gd, A.row0, A.row1, A.nboff), stg, mbar);
          }
          if (q.diag) {
            if (act) {
              double *dst = A.pdiag + (size_t)rc.x * 9;
#pragma unroll
              for (int i = 0; i < 9; ++i) dst[i] = (double)y[i];
            }
            continue;
          }
          // the transposed product to the block's slot (column order)
          if (act) store_transposed(A, rc.z, t);
          const int row = rc.x;
          // a group inside the open row (most groups: a row has hundreds of
          // blocks): every lane adds its product to its own FP64 running sum
          if (cur_row >= 0 && __all_sync(0xffffffffu, !act || row == cur_row)) {
            if (act)
#pragma unroll
              for (int j = 0; j < 9; ++j) lacc[j] += (double)y[j];
            continue;
          }
          // a row boundary: the lanes' running sums join the open row's sum,
          // then a segmented scan of the group's products (rows non-decreasing
          // in lane order; inactive lanes carry distinct negative rows)
          fold_lanes();
          segment_scan(row, y, lane);
          const int rnext = __shfl_down_sync(0xffffffffu, row, 1);
          const bool end = act && (lane == q.n - 1 || rnext != row);
          unsigned ends = __ballot_sync(0xffffffffu, end);
          int seg_first = 0;  // first lane of the segment ending at e
          while (ends) {
            const int e = __ffs(ends) - 1;
            ends &= ends - 1;
            const int re = __shfl_sync(0xffffffffu, row, e);
            double sv = 0.;
#pragma unroll
            for (int j = 0; j < 9; ++j) {
              const float tv = __shfl_sync(0xffffffffu, y[j], e);
              if (lane == j) sv = (double)tv;
            }
            if (re == cur_row) {
              racc += sv;
            } else {
              flush();
              // a segment starts the row unless it is the chunk's first and
              // the row began before the chunk
              cur_head = cur_row >= 0 || seg_first > 0 || q.boff + seg_first == (long long)__ldg(A.firstN + re);
              cur_row = re;
              racc = sv;
            }
            seg_first = e + 1;
          }
        }
        if (!ok) break;
        fold_lanes();
        flush();
        // the chunk's share of d^T A d, summed over its lanes in a fixed order
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) pdq += __shfl_xor_sync(0xffffffffu, pdq, o);
        if (lane == 0) A.pdqc[c] = pdq;
        c = cn;
        cn = c < nch ? grab() : nch;
      }
      __syncwarp();
      if (!ok) {
        // a copy that never completed: record it, give it one more bounded
        // wait, and leave at the grid barrier below
        if (lane == 0) atomicOr(A.err, 2);
        stage_wait(A, mbar, parity);
      }
    }

    if (!bar.sync(!ok)) return;
    double edtAdk;
    {
      // d^T A d: every CTA sums the chunks' shares in the same fixed order
      // (thread t takes chunks t, t + P32_T, ...; then a butterfly per warp
      // and the warps in order)
      double v = 0.;
      for (long long i = threadIdx.x; i < nch; i += P32_T) v += __ldcg(A.pdqc + i);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) sh[warp] = v;
      __syncthreads();
      double t = 0.;
      for (int w = 0; w < P32_W; ++w) t += sh[w];
      edtAdk = t;
    }
    double alpha;
    if (fabs(erthk) < 1.e-20 || fabs(erthk) > 1.e20)
      alpha = 0.;
    else
      alpha = erthk / edtAdk;
    // ---- phase 2
    double p2[3] = {0., 0., 0.};
    if constexpr (!CO) {
      for (int row = row_a; row < A.row1; row += nrw) {
        const size_t i = (size_t)row * 9 + (lane < 9 ? lane : 0);
        double r1v = 0., hv = 0.;
        const double q = row_q32(A, row, gd, ch, lane);
        if (lane < 9) {
          hv = __ldcg(A.h + i);
          const double dk = __ldcg(dcur + i);
          A.x[i] = A.x[i] + alpha * dk;
          const double dr = alpha * q;
          r1v = A.r[i] - dr;
          p2[0] += dr * dr;
        }
        const double *C = A.Cinv + (size_t)row * 81;
        double h1v = 0.;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const double rc = __shfl_sync(0xffffffffu, r1v, c);
          if (lane < 9) h1v += __ldg(C + lane * 9 + c) * rc;
        }
        if (lane < 9) {
          A.r[i] = r1v;
          A.h[i] = h1v;
          p2[1] += r1v * (h1v - hv);
          p2[2] += r1v * h1v;
        }
      }
    } else {
      __shared__ double shr[P32_W][CO_M + 1];
      __shared__ double shz[CO_M];
      // 2a: rows in any order, taken from a counter (the rows of high index,
      // with the longest runs of transposed products, first); each row's
      // results go to its own slots, so nothing depends on which warp took it
      // Every load of a row that does not depend on q is issued before the
      // row's walk: lanes 0..8 hold row `lane` of C_k, lanes 16..25 column
      // `lane - 16` of P_k (9 doubles a lane either way).
      const bool cl = lane < 9, pl = lane >= 16 && lane < 16 + CO_M;
      // one row; returns lanes 16 .. 25 the restriction, lane 31 (all lanes)
      // the share of dr^2 in d2
      auto take_row = [&](int row, double &d2) -> double {
        const size_t i = (size_t)row * 9 + (cl ? lane : 0);
        double cp[9];
        {
          const double *C = A.Cinv + (size_t)row * 81 + (cl ? lane * 9 : 0);
          const double *Pk = A.P + (size_t)row * (9 * CO_M) + (pl ? lane - 16 : 0);
#pragma unroll
          for (int c = 0; c < 9; ++c) cp[c] = cl ? __ldg(C + c) : (pl ? __ldg(Pk + c * CO_M) : 0.);
        }
        double dk = 0., xv = 0., rv = 0.;
        if (cl) {
          dk = __ldcg(dcur + i);
          xv = __ldcg(A.x + i);
          rv = __ldcg(A.r + i);
        }
        const double q = row_q32(A, row, gd, ch, lane);
        double r1v = 0.;
        d2 = 0.;
        if (cl) {
          A.x[i] = xv + alpha * dk;
          const double dr = alpha * q;
          r1v = rv - dr;
          d2 = dr * dr;
        }
        double acc = 0.;  // lanes 0..8: h_j; lanes 16..25: the restriction
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          const double rc = __shfl_sync(0xffffffffu, r1v, c);
          acc += cp[c] * rc;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, o);
        if (cl) {
          A.r[i] = r1v;
          A.hj[i] = acc;
        }
        return acc;
      };
      if constexpr (SMALL) {
        // an aggregate's rows by its CTA's warps (warp w: rows w, w + P32_W,
        // ...), then its restriction and share of dr^2, the warps in order
        for (int a = blockIdx.x; a < A.nagg; a += G) {
          const int t0 = A.agg_off[a], t1 = A.agg_off[a + 1];
          double v = 0.;  // lanes 16 .. 25, and 31
          for (int t = t0 + warp; t < t1; t += P32_W) {
            double d2;
            const double acc = take_row(A.agg_rows[t], d2);
            if (pl) v += acc;
            if (lane == 31) v += d2;
          }
          if (pl) shr[warp][lane - 16] = v;
          if (lane == 31) shr[warp][CO_M] = v;
          __syncthreads();
          if (threadIdx.x <= CO_M) {
            double sum = 0.;
            for (int w = 0; w < P32_W; ++w) sum += shr[w][threadIdx.x];
            if (threadIdx.x < CO_M)
              A.rc[a * CO_M + threadIdx.x] = sum;
            else
              A.rowc[a] = sum;  // joins the aggregates' sum in 2b, in the one-warp form's order
          }
          __syncthreads();
        }
      } else {
        const int nrows = A.row1 - A.row0;
        auto grab_row = [&]() -> int {
          unsigned t = 0;
          if (lane == 0) t = atomicAdd(A.ctr + 1, 1u);
          return (int)__shfl_sync(0xffffffffu, t, 0);
        };
        for (int t = grab_row(); t < nrows;) {
          const int row = A.row1 - 1 - t;
          const int tn = grab_row();  // the next row, taken one ahead
          double d2;
          const double acc = take_row(row, d2);
          if (pl) A.rowc[(size_t)row * RC_S + lane - 16] = acc;
          if (lane == 31) A.rowc[(size_t)row * RC_S + CO_M] = d2;
          t = tn;
        }
        if (!bar.sync()) return;
        // 2a': per aggregate, its rows' restrictions and shares of dr^2 in a
        // fixed order (warp w: rows w, w + P32_W, ...; then the warps in order)
        for (int a = blockIdx.x; a < A.nagg; a += G) {
          const int t0 = A.agg_off[a], t1 = A.agg_off[a + 1];
          double v = 0.;
          if (lane <= CO_M)
            for (int t = t0 + warp; t < t1; t += P32_W) v += __ldcg(A.rowc + (size_t)A.agg_rows[t] * RC_S + lane);
          if (lane <= CO_M) shr[warp][lane] = v;
          __syncthreads();
          if (threadIdx.x <= CO_M) {
            double sum = 0.;
            for (int w = 0; w < P32_W; ++w) sum += shr[w][threadIdx.x];
            if (threadIdx.x < CO_M)
              A.rc[a * CO_M + threadIdx.x] = sum;
            else
              p2[0] += sum;
          }
          __syncthreads();
        }
      }
      if (!bar.sync()) return;
      // z of an aggregate: its rows of A_c^-1 with the restrictions, a warp's share
      auto z_share = [&](int a) -> double {
        double z[CO_M];
#pragma unroll
        for (int j = 0; j < CO_M; ++j) z[j] = 0.;
        for (int i = threadIdx.x; i < A.nc; i += P32_T) {
          const double rv = __ldcg(A.rc + i);
#pragma unroll
          for (int j = 0; j < CO_M; ++j) z[j] += __ldg(A.Ainv + (size_t)(a * CO_M + j) * A.nc + i) * rv;
        }
        return butterfly_scatter<CO_M>(z, lane);
      };
      if constexpr (SMALL) {
        // the g0 CTAs of the one-warp form, whose shares of the sums they add:
        // ZB aggregates at a time, a warp's rows of them in threes (lanes 9 s
        // + j), their terms added in the rows' order
        constexpr int ZB = 4;
        __shared__ double shr4[ZB][P32_W][CO_M + 1], shz4[ZB][CO_M];
        const int G2 = A.g0, sub = lane / 9, jr = lane - 9 * sub;
        for (int a0 = (int)blockIdx.x < G2 ? (int)blockIdx.x : A.nagg; a0 < A.nagg; a0 += ZB * G2) {
#pragma unroll 1
          for (int b = 0; b < ZB && a0 + b * G2 < A.nagg; ++b) {
            const double zs = z_share(a0 + b * G2);
            if ((lane & 1) == 0 && lane < 2 * CO_M) shr4[b][warp][lane >> 1] = zs;
          }
          __syncthreads();
          if (threadIdx.x < ZB * CO_M) {
            const int b = threadIdx.x / CO_M, j = threadIdx.x - CO_M * b;
            if (a0 + b * G2 < A.nagg) {
              double sum = 0.;
              for (int w = 0; w < P32_W; ++w) sum += shr4[b][w][j];
              shz4[b][j] = sum;
            }
          }
          if (threadIdx.x == CO_M)
            for (int b = 0; b < ZB && a0 + b * G2 < A.nagg; ++b) p2[0] += __ldcg(A.rowc + a0 + b * G2);
          __syncthreads();
          // a place in the warp's list of rows: aggregate b, row t of it
          int b = 0, t = __ldg(A.agg_off + a0) + warp, t1 = __ldg(A.agg_off + a0 + 1);
          auto settle = [&]() {
            while (t >= t1 && ++b < ZB && a0 + b * G2 < A.nagg) {
              t = __ldg(A.agg_off + a0 + b * G2) + warp;
              t1 = __ldg(A.agg_off + a0 + b * G2 + 1);
            }
          };
          settle();
          for (int s = 0; s < sub && t < t1; ++s) {
            t += P32_W;
            settle();
          }
          while (__any_sync(0xffffffffu, t < t1)) {
            const bool act = t < t1 && sub < 3;
            double r1v = 0., dh = 0., h1v = 0.;
            if (act) {
              const int row = __ldg(A.agg_rows + t);
              const size_t i = (size_t)row * 9 + jr;
              const double *Pk = A.P + (size_t)row * (9 * CO_M) + jr * CO_M;
              h1v = __ldcg(A.hj + i);
#pragma unroll
              for (int j = 0; j < CO_M; ++j) h1v += __ldg(Pk + j) * shz4[b][j];
              const double hv = __ldcg(A.h + i);
              r1v = __ldcg(A.r + i);
              dh = h1v - hv;
              A.h[i] = h1v;
            }
#pragma unroll
            for (int s = 0; s < 3; ++s) {
              const int src = lane < 9 ? 9 * s + lane : lane;
              const double rs = __shfl_sync(0xffffffffu, r1v, src), ds = __shfl_sync(0xffffffffu, dh, src),
                           hs = __shfl_sync(0xffffffffu, h1v, src);
              if (lane < 9) {
                p2[1] += rs * ds;
                p2[2] += rs * hs;
              }
            }
            for (int s = 0; s < 3 && t < t1; ++s) {
              t += P32_W;
              settle();
            }
          }
        }
      } else {
        for (int a = blockIdx.x; a < A.nagg; a += G) {
          {
            const double zs = z_share(a);
            if ((lane & 1) == 0 && lane < 2 * CO_M) shr[warp][lane >> 1] = zs;
          }
          __syncthreads();
          if (threadIdx.x < CO_M) {
            double sum = 0.;
            for (int w = 0; w < P32_W; ++w) sum += shr[w][threadIdx.x];
            shz[threadIdx.x] = sum;
          }
          __syncthreads();
          const int t0 = A.agg_off[a], t1 = A.agg_off[a + 1];
          for (int t = t0 + warp; t < t1; t += P32_W) {
            const int row = A.agg_rows[t];
            if (lane < 9) {
              const size_t i = (size_t)row * 9 + lane;
              const double *Pk = A.P + (size_t)row * (9 * CO_M) + lane * CO_M;
              double h1v = __ldcg(A.hj + i);
#pragma unroll
              for (int j = 0; j < CO_M; ++j) h1v += __ldg(Pk + j) * shz[j];
              const double hv = __ldcg(A.h + i), r1v = __ldcg(A.r + i);
              p2[1] += r1v * (h1v - hv);
              p2[2] += r1v * h1v;
              A.h[i] = h1v;
            }
          }
          __syncthreads();
        }
      }
    }
    if (!exchange_sum<3, P32_W>(bar, A.red2, p2, X2)) return;
    const double(&g3)[3] = p2;
    const double meandr = g3[0], er1th1 = g3[1];
    if (k == 0) meandr0 = meandr;
    const bool finite = isfinite(g3[0]) && isfinite(g3[2]);
    const bool improved = (A.mode == 1 && finite) || meandr < meandrold;
    if (improved) {
      meandrold = meandr;
      for (int row = row_a; row < A.row1; row += nrw)
        if (lane < 9) A.xbest[(size_t)row * 9 + lane] = __ldcg(A.x + (size_t)row * 9 + lane);
    }
    if (A.mode == 0 && meandr * 1.e5 < meandr0) break;
    if (A.mode == 1 && !finite) break;
    if (A.mode == 1 && g3[2] <= A.tol2 * erthk0) {
      converged = true;
      break;
    }
    double beta = fabs(er1th1) < 1.e-10 ? 0. : er1th1 / erthk;
    if (beta < 0.) beta = 0.;
    beta_prev = beta;
    erthk = g3[2];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.iters[0] = k < A.msize ? k + 1 : A.msize;
    A.iters[1] = converged ? 1 : 0;
  }
}

// Preconditioner C_k = S_kk^-1 (rbacore.cpp:1839-1846) and the start
// vectors: r = b, h = C r, d^(-1) = 0, x = 0, best = b.  One warp per camera
// (lu_inverse9_warp): a thread per camera with its factor in local memory
// took 76 us for 12 cameras and 145 us for 1,370, now 15 and 20 us.
// PLAIN: the drop-in form, whose numerics are lu_inverse9's.
constexpr int SETUP_W = 2;  // warps per CTA: few cameras are spread over the SMs
template <bool PLAIN>
__global__ void __launch_bounds__(32 * SETUP_W) k_pcg_setup(DevLSA L, PcgWork W) {
  const int k = blockIdx.x * SETUP_W + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= L.nimg) return;
  double *C = W.Cinv + (size_t)k * 81;
  const size_t o = (size_t)k * 9 + lane;
  if (lane < 9) W.d[o] = 0.;
  if (k < L.begini) {
    if (lane < 9) W.r[o] = W.h[o] = W.x[o] = W.xbest[o] = 0.;
    return;
  }
  const int np = L.camparv[k + 1] - L.camparv[k];
  double row[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) row[c] = lane < 9 ? blk_at(L, (size_t)k, lane * 9 + c) : 0.;
  const double rv = lane < 9 ? L.rhs[o] : 0.;
  lu_inverse9_warp<PLAIN>(np, row, C, lane);
  __syncwarp();
  double s = 0.;
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    const double rc = __shfl_sync(0xffffffffu, rv, c);
    if (lane < 9) s += C[lane * 9 + c] * rc;
  }
  if (lane < 9) {
    W.r[o] = rv;
    W.h[o] = s;
    W.x[o] = 0.;
    W.xbest[o] = rv;
  }
}

// Test of lu_inverse9_warp<true>: matrix blockIdx.x inverted by one thread and
// by the warp.
__global__ void k_lu_both(const double *A, int np, double *by_thread, double *by_warp) {
  const int lane = threadIdx.x;
  const double *a = A + (size_t)blockIdx.x * 81;
  if (lane == 0) lu_inverse9(np, a, by_thread + (size_t)blockIdx.x * 81);
  __syncwarp();
  double row[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) row[c] = lane < 9 ? a[lane * 9 + c] : 0.;
  lu_inverse9_warp<true>(np, row, by_warp + (size_t)blockIdx.x * 81, lane);
}

}  // namespace

void lu_inverse9_both(const double *A, int count, int np, double *by_thread, double *by_warp, cudaStream_t s) {
  k_lu_both<<<count, 32, 0, s>>>(A, np, by_thread, by_warp);
  RPBA_CUDA_CHECK(cudaGetLastError());
}

// the blocks and stages live in dynamic shared memory (FP64 resident 212,992 B,
// streamed 213,472 B)
void pcg_set_smem() {
  auto set = [](auto k, size_t bytes) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  set(k_pcg<false, PCG_RESIDENT>, pcg_smem_bytes<PCG_RESIDENT>());
  set(k_pcg<true, PCG_RESIDENT>, pcg_smem_bytes<PCG_RESIDENT>());
  set(k_pcg<false, PCG_STREAMED>, pcg_smem_bytes<PCG_STREAMED>());
  set(k_pcg<true, PCG_STREAMED>, pcg_smem_bytes<PCG_STREAMED>());
  set(k_pcg32<false, false>, P32_SMEM);
  set(k_pcg32<true, false>, P32_SMEM);
  set(k_pcg32<false, true>, P32_SMEM);
  set(k_pcg32<true, true>, P32_SMEM);
}

// Groups of 32 blocks per phase-1 chunk of the FP32 PCG: small enough that
// the warps finish together, large enough that a chunk's fixed work (its
// first segmented scan, its sums) stays small (city workload, phase 1 with
// its barrier: 2 groups 377 us, 4 groups 365 us, 8 groups 379 us).
constexpr int PCG32_CHUNK = 4;

// Bytes of blocks from which on the FP64 streamed form reads them with an
// evict-first hint.  With products and index, a quarter on top, the system
// reaches the 126 MB of L2 at 100 MB of blocks, and the hint keeps the products
// there.  An iteration without and with it, by size of the blocks: 24 MB 26.6
// and 26.9 us, 76 MB 52.3 and 52.4, 82 MB 54.8 and 53.4, 123 MB 75.7 and 68.7,
// 177 MB 98.8 and 90.4, 241 MB 126.7 and 120.4.
constexpr double STREAM_ONCE_BYTES = 6.4e7;

int pcg_max_grid(int device) {
  int nsm = 0, per = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  pcg_set_smem();
  per = 1 << 30;
  auto fit = [&](auto k, int threads, size_t smem) {
    int p = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, k, threads, smem);
    per = std::min(per, p);
  };
  fit(k_pcg<false, PCG_RESIDENT>, P64_T, pcg_smem_bytes<PCG_RESIDENT>());
  fit(k_pcg<true, PCG_RESIDENT>, P64_T, pcg_smem_bytes<PCG_RESIDENT>());
  fit(k_pcg<false, PCG_STREAMED>, P64_T, pcg_smem_bytes<PCG_STREAMED>());
  fit(k_pcg<true, PCG_STREAMED>, P64_T, pcg_smem_bytes<PCG_STREAMED>());
  fit(k_pcg<false, PCG_GATHERED>, P64_T, 0);
  fit(k_pcg<true, PCG_GATHERED>, P64_T, 0);
  fit(k_pcg32<false, false>, P32_T, P32_SMEM);
  fit(k_pcg32<true, false>, P32_T, P32_SMEM);
  fit(k_pcg32<false, true>, P32_T, P32_SMEM);
  fit(k_pcg32<true, true>, P32_T, P32_SMEM);
  if (per < 1) per = 1;
  return std::min(nsm * per, XMAXG - 1);
}

// CTAs of the FP64 form: an item a warp
static int grid64(int nitems, int grid) {
  return std::max(1, std::min((nitems + P64_W - 1) / P64_W, grid));
}
// its groups of 32 blocks, see group64
static long long groups64(const DevLSA &L) { return (L.nimg - L.begini + 31) / 32 + (L.nboff + 31ll) / 32; }

bool pcg_blocks_stay(const DevLSA &L, int form, int grid) {
  if (form == PCG_STREAMED && !L.blocks32) return groups64(L) <= (long long)P1S_N * grid64(L.nitems, grid);
  return form == PCG_RESIDENT;
}

int pcg_resident_items(int grid) { return P1_SLOTS * P64_W * grid; }

// barrier word (and padding), then the CTAs' sums of the two exchanges
size_t pcg_bar_bytes() { return 16 + 4 * (size_t)XMAXG * sizeof(double); }

// Returns 0; throws CudaError on launch errors.  The iteration count is
// left in W.iters.
int pcg_prepare(const DevLSA &L, const PcgWork &W, int mode, const float *weights, const CoarseWork *coarse,
                cudaStream_t s) {
  const bool co = coarse && coarse->nagg > 0;
  const int g = (L.nimg + SETUP_W - 1) / SETUP_W;
  if (weights)
    learned_pcg_setup(L, W, weights, s);
  else if (mode == 1 || co)
    k_pcg_setup<false><<<g, 32 * SETUP_W, 0, s>>>(L, W);
  else
    k_pcg_setup<true><<<g, 32 * SETUP_W, 0, s>>>(L, W);
  if (co) coarse_apply(L, *coarse, W.r, W.h, s);
  RPBA_CUDA_CHECK(cudaGetLastError());
  return co ? 3 : 1;
}

int pcg_iterate(const DevLSA &L, const PcgWork &W, int msize, int grid, cudaStream_t s, int mode, double tol,
                const CoarseWork *coarse) {
  const bool co = coarse && coarse->nagg > 0;
  const int nrows = L.nimg - L.begini;
  if (nrows <= 0) return 0;
  int g, g0 = 0;
  bool small32 = false;
  if (L.blocks32) {
    // FP32 form: groups of 32 blocks (the diagonal blocks of the system's
    // rows, then the off-diagonal blocks), at least one group per warp
    const long long ng = (nrows + GB - 1) / GB + ((long long)L.nboff + GB - 1) / GB;
    // at least one group per warp (g0); a system of at most one group per
    // warp of the whole grid is spread further: a chunk, and with the coarse
    // space an aggregate, per CTA (a barrier over 148 CTAs instead of 58 costs
    // 500 cycles, a second chunk or aggregate on an SM thousands)
    g0 = (int)std::min<long long>((ng + P32_W - 1) / P32_W, grid);
    small32 = ng <= (long long)grid * P32_W && PCG32_CHUNK == 4 && W.force_form <= PCG_RESIDENT;
    g = g0;
    if (small32) g = (int)std::max<long long>(std::max<long long>(g, (ng + 3) / 4), co ? coarse->nagg : 0);
    g = (int)std::min<long long>(g, grid);
  } else {
    g = grid64(L.nitems, grid);
  }
  if (g > grid) g = grid;
  if (g < 1) g = 1;
  PcgArgs A;
  A.blocks = L.blocks32 ? (const void *)L.blocks32 : (const void *)L.blocks;
  A.row_item_off = L.row_item_off;
  A.item_rec = L.item_rec;
  A.ent = L.ent;
  A.prod = W.prod;
  A.tpart = L.tpart;
  A.bidx = L.bidx;
  A.firstN = L.firstN;
  A.firstT = L.firstT;
  A.nboff = L.nboff;
  A.d32 = W.d32;
  A.pdiag = W.pdiag;
  A.prow = W.prow;
  A.pw = W.pw;
  A.pdqc = W.pdqc;
  A.ctr = W.ctr;
  A.rowc = W.rowc;
  A.chunk = PCG32_CHUNK;
  A.g0 = g0;
  A.Cinv = W.Cinv;
  A.r = W.r;
  A.h = W.h;
  A.x = W.x;
  A.xbest = W.xbest;
  A.D0 = W.q;
  A.D1 = W.d;
  A.part = W.part;
  A.bar = W.bar;
  A.red1 = (double *)(W.bar + 4);
  A.red2 = A.red1 + XMAXG;
  A.err = L.err;
  A.iters = W.iters;
  A.bar_extra = L.bar_extra;
  A.bar_ns = L.bar_timeout_ns ? L.bar_timeout_ns : BAR_TIMEOUT_NS;
  A.tx_extra = L.wait_fault == 1 ? 16u : 0u;
  A.row0 = L.begini;
  A.row1 = L.nimg;
  A.nitems = L.nitems;
  A.stream_once = ((double)nrows + L.nboff) * 648. > STREAM_ONCE_BYTES;
  A.msize = msize;
  A.mode = mode;
  A.tol2 = tol * tol;
  A.nagg = co ? coarse->nagg : 0;
  A.nc = co ? coarse->nc : 0;
  A.agg_off = co ? coarse->agg_off : nullptr;
  A.agg_rows = co ? coarse->agg_rows : nullptr;
  A.P = co ? coarse->P : nullptr;
  A.Ainv = co ? coarse->Ainv : nullptr;
  A.rc = co ? coarse->rc : nullptr;
  A.hj = co ? coarse->hj : nullptr;
  RPBA_CUDA_CHECK(cudaMemsetAsync(W.bar, 0, 4 * sizeof(unsigned), s));
  void *args[] = {&A};
  const void *fn;
  size_t smem;
  int nthreads, form;
  if (L.blocks32) {
    fn = co ? (small32 ? (const void *)k_pcg32<true, true> : (const void *)k_pcg32<true, false>)
            : (small32 ? (const void *)k_pcg32<false, true> : (const void *)k_pcg32<false, false>);
    smem = P32_SMEM;
    nthreads = P32_T;
    form = small32 ? PCG_RESIDENT : PCG_STREAMED;
  } else {
    form = L.item_words == 4 ? PCG_RESIDENT : (W.prod ? PCG_STREAMED : PCG_GATHERED);
    if (form == PCG_RESIDENT) {
      fn = co ? (const void *)k_pcg<true, PCG_RESIDENT> : (const void *)k_pcg<false, PCG_RESIDENT>;
      smem = pcg_smem_bytes<PCG_RESIDENT>();
    } else if (form == PCG_STREAMED) {
      fn = co ? (const void *)k_pcg<true, PCG_STREAMED> : (const void *)k_pcg<false, PCG_STREAMED>;
      smem = pcg_smem_bytes<PCG_STREAMED>();
    } else {
      fn = co ? (const void *)k_pcg<true, PCG_GATHERED> : (const void *)k_pcg<false, PCG_GATHERED>;
      smem = 0;
    }
    nthreads = P64_T;
  }
  pcg_set_smem();
  RPBA_CUDA_CHECK(cudaLaunchCooperativeKernel(fn, dim3(g), dim3(nthreads), args, smem, s));
  return form;
}

}  // namespace rpba
