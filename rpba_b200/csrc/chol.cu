// chol.cu -- tiled FP64 Cholesky factorisation of symmetric positive definite
// matrices held as 64 x 64 tiles, in one cooperative launch, with the tile
// products on the FP64 tensor cores (mma.sync m8n8k4 f64; sm_100a has no
// FP64 kind of tcgen05.mma).
//
// Storage: the lower triangle in tiles, row by row; tile row I holds the
// tiles of columns fcol[I] .. I, with fcol nondecreasing (an envelope: a
// dense matrix has fcol = 0).  A Cholesky factor keeps the envelope of its
// matrix, so L overwrites A in place.  hrow[J] is the last tile row whose
// envelope reaches column J.
//
// Right-looking, per tile column J:
//   P  the diagonal tile is factored and inverted: L_JJ and L_JJ^-1
//      (Linv[J]), potrf_tile;
//   T  every tile below it: L_IJ = A_IJ L_JJ^-T, a tile product;
//   U  the trailing tiles: A_IK -= L_IJ L_KJ^T for J < K <= I <= hrow[J].
// The chain P(J), T of tile (J + 1, J), U of tile (J + 1, J + 1), P(J + 1)
// bounds the launch, so CTA 0 runs that chain alone, the tiles passing
// through its shared memory, and the other CTAs the rest of T and U of
// column J meanwhile (dealt round robin).  Two bounded grid barriers a
// column: between the others' T and U (CTA 0 arrives once its tile of T is
// stored and does not wait), and at the column's end.  A non-positive pivot
// sets bit 4 of the error word.
// Measured on the aerial system (26,991 unknowns, 422 tile columns, band of
// 21 to 33 tiles): 13.9 ms with every CTA in step (two full barriers a
// column, CTA 0's tile reloaded in each phase), 10.6 ms so.
//
// For a dense matrix the same launch can go on to the inverse:
//   X  = L^-1, right-looking by tile rows: X_Ij = Linv_I R_Ij (j <= I), then
//        R_Kj -= L_KI X_Ij for K > I;
//   A^-1 = X^T X, one output tile per work item, both triangles written.
#include "gridsync.cuh"
#include "internal.h"

namespace rpba {

namespace {

constexpr int CT = 64;                  // tile edge
constexpr int CLD = 68;                 // shared leading dimension: conflict-free fragment loads
constexpr int CTH = 512;                // threads per CTA (16 warps)
constexpr int TS = CT * CT;             // doubles per stored tile
static_assert(CTH == 8 * CT, "tile loads: eight lanes a row");
constexpr int NF = 4;                   // 8 x 8 fragments per warp
constexpr size_t CSMEM = (2 * CT * CLD + 4 * CT) * sizeof(double);  // two tiles + partials

struct Tiles {
  double *L;               // tile storage (row major inside a tile, ld 64)
  const long long *toff;   // [nt] first tile of row I
  const int *fcol;         // [nt] first tile column of row I
  const int *hrow;         // [nt] last tile row reaching column J
  double *Linv;            // [nt][TS] inverses of the diagonal tiles
  double *X;               // dense inverse only: [nt(nt+1)/2][TS] L^-1, lower tiles
  double *Ainv;            // dense inverse only: [nt(nt+1)/2][TS] A^-1, lower tiles
  int nt;
  int want_inverse;
  unsigned *bar;
  int *err;
  unsigned bar_extra;  // arrivals that never come (test hook)
  unsigned long long bar_ns;
};

__device__ __forceinline__ double *tile_at(const Tiles &T, int I, int J) {
  return T.L + (size_t)(T.toff[I] + (J - T.fcol[I])) * TS;
}
__device__ __forceinline__ size_t tri(int I, int J) { return (size_t)I * (I + 1) / 2 + J; }

// D (8x8, two per thread) += A (8x4, one per thread) * B (4x8, one per thread)
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// acc (warp w: rows 8 (w % 8) .. + 7, columns 32 (w / 8) .. + 31, 4
// fragments of 2) += sA sB^T over k = 0 .. 63; sA, sB in shared memory with
// ld CLD.
__device__ __forceinline__ int frag_row() { return 8 * ((threadIdx.x >> 5) & 7) + ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int frag_col() { return 32 * (threadIdx.x >> 8) + 2 * (threadIdx.x & 3); }
__device__ __forceinline__ void gemm_nt(const double *sA, const double *sB, double (&acc)[NF][2]) {
  const int lane = threadIdx.x & 31, t = lane & 3;
  const double *pa = sA + frag_row() * CLD + t;
  const double *pb = sB + (32 * (threadIdx.x >> 8) + (lane >> 2)) * CLD + t;
#pragma unroll 4
  for (int kk = 0; kk < CT / 4; ++kk) {
    const double a = pa[4 * kk];
#pragma unroll
    for (int j = 0; j < NF; ++j) dmma(acc[j][0], acc[j][1], a, pb[8 * j * CLD + 4 * kk]);
  }
}

// Global tile (ld 64) -> shared (ld CLD), optionally transposed: every
// thread's four 16-byte loads are issued before its first store.
__device__ __forceinline__ void load_tile(double *s, const double *g, bool trans) {
  const int i = threadIdx.x >> 3, j0 = 2 * (threadIdx.x & 7);
  double2 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = __ldcg((const double2 *)(g + i * CT + 16 * q + j0));
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = 16 * q + j0;
    if (trans) {
      s[j * CLD + i] = v[q].x;
      s[(j + 1) * CLD + i] = v[q].y;
    } else {
      *(double2 *)(s + i * CLD + j) = v[q];
    }
  }
}

// Tile update gt -= acc (fragment positions): the old values are loaded
// before any is written back.
__device__ __forceinline__ void sub_frag(double *gt, const double (&acc)[NF][2]) {
  double *g = gt + frag_row() * CT + frag_col();
  double2 old[NF];
#pragma unroll
  for (int j = 0; j < NF; ++j) old[j] = __ldcg((const double2 *)(g + 8 * j));
#pragma unroll
  for (int j = 0; j < NF; ++j) *(double2 *)(g + 8 * j) = make_double2(old[j].x - acc[j][0], old[j].y - acc[j][1]);
}
// The same with the result left in shared memory (ld CT + 1).
__device__ __forceinline__ void sub_frag_to(const double *gt, const double (&acc)[NF][2], double *s) {
  const double *g = gt + frag_row() * CT + frag_col();
  double *d = s + frag_row() * (CT + 1) + frag_col();
  double2 old[NF];
#pragma unroll
  for (int j = 0; j < NF; ++j) old[j] = __ldcg((const double2 *)(g + 8 * j));
#pragma unroll
  for (int j = 0; j < NF; ++j) {
    d[8 * j] = old[j].x - acc[j][0];
    d[8 * j + 1] = old[j].y - acc[j][1];
  }
}
__device__ __forceinline__ void store_frag(double *gt, const double (&acc)[NF][2]) {
  double *g = gt + frag_row() * CT + frag_col();
#pragma unroll
  for (int j = 0; j < NF; ++j) *(double2 *)(g + 8 * j) = make_double2(acc[j][0], acc[j][1]);
}

// Factor the diagonal tile in s (lower triangle, ld PLD) and write L_JJ and
// L_JJ^-1, with all threads of the CTA.
//
// The chain of the 64 pivots (a square root, a reciprocal, the next pivot's
// update: about 160 cycles each) bounds the whole factorisation, so warp 0
// runs that chain and as little else as it can: the 8 x 8 diagonal block of
// a panel, held whole in every lane's registers (no exchange between the
// pivots), then only the next block's eight rows and its update.  Meanwhile
// warps 1-7 solve the panel's other rows and apply the panel to the columns
// past it, and warps 8-15 form the panel's rows of the inverse; one block
// barrier a panel.  Every entry takes its updates in column order, and every
// inverse entry its four partial sums (terms mm = c + q, c + q + 4, ... in
// order, then (p0 + p1) + (p2 + p3)), as the unblocked column loop takes
// them, so the result does not depend on the distribution.
// A tile takes 31,800 cycles (16.5 us; 125,000 with one warp factoring panels
// and the inverse formed after them).
// s, si: two shared tiles (ld PLD); pp: CT doubles (reciprocal pivots).
constexpr int PLD = CT + 1, PW = 8;

// Rows [r0, r0 + PW) of the inverse of the factored tile, by warps 8 .. 15:
// four lanes per column c, lane q its partial sum q.  The terms of earlier
// blocks' rows first (eight rows' sums side by side), then the block's own
// rows one after the other.
__device__ __forceinline__ void inverse_block(int r0, const double *s, double *si, const double *pp) {
  const int lane = threadIdx.x & 31, c = ((threadIdx.x >> 5) - 8) * 8 + (lane >> 2), q = lane & 3;
  double u[PW];
#pragma unroll
  for (int r = 0; r < PW; ++r) u[r] = 0.;
  const double *sr = s + r0 * PLD, *sc = si + c;
#pragma unroll 2
  for (int mm = c + q; mm < r0; mm += 4) {
    const double x = sc[mm * PLD];
#pragma unroll
    for (int r = 0; r < PW; ++r) u[r] += sr[r * PLD + mm] * x;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < PW; ++r) {
    const int i = r0 + r;
    const double p2 = u[r] + __shfl_xor_sync(0xffffffffu, u[r], 1);
    const double p4 = p2 + __shfl_xor_sync(0xffffffffu, p2, 2);
    const double rdi = pp[i];
    const double z = c < i ? -p4 * rdi : (c == i ? rdi : 0.);
    si[i * PLD + c] = z;  // the column's four lanes write the same value
    // the term mm = i of the block's later rows, in its partial sum
    const double zq = c <= i && ((i - c) & 3) == q ? z : 0.;
#pragma unroll
    for (int t = r + 1; t < PW; ++t) u[t] += sr[t * PLD + i] * zq;
  }
  __syncwarp();
}

__device__ __forceinline__ void load_potrf_tile(const double *gtile, double *s) {
  const int t = threadIdx.x;
  double2 v[TS / CTH / 2];
#pragma unroll
  for (int q = 0; q < TS / CTH / 2; ++q) v[q] = __ldcg((const double2 *)gtile + t + q * CTH);
#pragma unroll
  for (int q = 0; q < TS / CTH / 2; ++q) {
    const int e = 2 * (t + q * CTH);
    s[(e >> 6) * PLD + (e & 63)] = v[q].x;
    s[(e >> 6) * PLD + (e & 63) + 1] = v[q].y;
  }
}

// x (a row's eight entries of a panel) solved by the panel's diagonal block:
// entry j takes the updates k = 0 .. j - 1 in order, then its pivot.
// (l: the block, ld PLD; rd: its reciprocal pivots)
__device__ __forceinline__ void panel_row_solve(double (&x)[PW], const double *rd, const double *l) {
#pragma unroll
  for (int k = 0; k < PW; ++k) {
    x[k] *= rd[k];
#pragma unroll
    for (int j = k + 1; j < PW; ++j) x[j] -= x[k] * l[j * PLD + k];
  }
}

__device__ void potrf_tile(double *gtile, double *ginv, int *err, double *s, double *si, double *pp) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  __syncthreads();
#pragma unroll 1
  for (int k0 = 0; k0 < CT; k0 += PW) {
    const int kp = k0 - PW;  // the previous panel
    if (w == 0) {
      if (k0 > 0) {
        // this block's rows of the previous panel (lane: row lane % 8), then
        // its diagonal block's update (lane: two entries of that row)
        const int i = k0 + (lane & 7);
        double x[PW];
#pragma unroll
        for (int j = 0; j < PW; ++j) x[j] = s[i * PLD + kp + j];
        panel_row_solve(x, pp + kp, s + kp * PLD + kp);
        __syncwarp();
        // (every store below is made by all the lanes that hold the value)
#pragma unroll
        for (int j = 0; j < PW; ++j) s[i * PLD + kp + j] = x[j];
        __syncwarp();
        asm volatile("bar.arrive 1, 256;" ::: "memory");
        const int j0 = k0 + 2 * (lane >> 3);
        double y0 = s[i * PLD + j0], y1 = s[i * PLD + j0 + 1];
#pragma unroll
        for (int k = 0; k < PW; ++k) {
          y0 -= x[k] * s[j0 * PLD + kp + k];
          y1 -= x[k] * s[(j0 + 1) * PLD + kp + k];
        }
        s[i * PLD + j0] = y0;
        s[i * PLD + j0 + 1] = y1;
        __syncwarp();
      }
      double d[PW][PW], rd[PW];  // the diagonal block (lower), its reciprocal pivots
#pragma unroll
      for (int i = 0; i < PW; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) d[i][j] = s[(k0 + i) * PLD + k0 + j];
      bool bad = false;
#pragma unroll
      for (int k = 0; k < PW; ++k) {
        const double p = d[k][k];
        bad = bad || !(p > 0.);
        const double dk = sqrt(p > 0. ? p : 1.), rdk = 1. / dk;
        rd[k] = rdk;
        d[k][k] = dk;
#pragma unroll
        for (int i = k + 1; i < PW; ++i) d[i][k] *= rdk;
#pragma unroll
        for (int j = k + 1; j < PW; ++j)
#pragma unroll
          for (int i = j; i < PW; ++i) d[i][j] -= d[i][k] * d[j][k];
      }
      if (bad && lane == 0) atomicOr(err, 4);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < PW; ++i) {
        pp[k0 + i] = rd[i];
#pragma unroll
        for (int j = 0; j <= i; ++j) s[(k0 + i) * PLD + k0 + j] = d[i][j];
      }
    } else if (k0 > 0) {
      if (w < 8) {
        // the previous panel's rows past this block (warps 1 and 2)
        const int i = k0 + PW + (w - 1) * 32 + lane;
        if (i < CT) {
          double x[PW];
#pragma unroll
          for (int j = 0; j < PW; ++j) x[j] = s[i * PLD + kp + j];
          panel_row_solve(x, pp + kp, s + kp * PLD + kp);
#pragma unroll
          for (int j = 0; j < PW; ++j) s[i * PLD + kp + j] = x[j];
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        // and its update of the columns j >= k0 (rows past this block):
        // lane: rows lane, lane + 32, the columns dealt to the seven warps
        double l[2][PW];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int k = 0; k < PW; ++k) l[h][k] = s[(lane + 32 * h) * PLD + kp + k];
#pragma unroll 2
        for (int j = k0 + w - 1; j < CT; j += 7) {
          double m[PW];
#pragma unroll
          for (int k = 0; k < PW; ++k) m[k] = s[j * PLD + kp + k];
          // (rows that take no update are computed and not stored: no branch
          // between the two rows' chains)
          double y[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) y[h] = s[(lane + 32 * h) * PLD + j];
#pragma unroll
          for (int k = 0; k < PW; ++k)
#pragma unroll
            for (int h = 0; h < 2; ++h) y[h] -= l[h][k] * m[k];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int row = lane + 32 * h;
            if (row >= j && row >= k0 + PW) s[row * PLD + j] = y[h];
          }
        }
      } else {
        inverse_block(kp, s, si, pp);
      }
    }
    __syncthreads();
  }
  if (w >= 8)
    inverse_block(CT - PW, s, si, pp);
  else
    for (int idx = t; idx < TS; idx += CTH / 2) {
      const int i = idx >> 6, j = idx & 63;
      gtile[idx] = j <= i ? s[i * PLD + j] : 0.;
    }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < TS / CTH; ++q) {
    const int idx = t + q * CTH;
    ginv[idx] = si[(idx >> 6) * PLD + (idx & 63)];
  }
  __syncthreads();
}

// k-th item of the lower triangle (bi >= bk) of an m x m tile triangle
__device__ __forceinline__ void tri_item(long long t, int &bi, int &bk) {
  int i = (int)((sqrt(8. * (double)t + 1.) - 1.) / 2.);
  while ((long long)(i + 1) * (i + 2) / 2 <= t) ++i;
  while ((long long)i * (i + 1) / 2 > t) --i;
  bi = i;
  bk = (int)(t - (long long)i * (i + 1) / 2);
}

__global__ void __launch_bounds__(CTH, 1) k_chol_tiles(Tiles T) {
  extern __shared__ __align__(16) double csm[];
  double *sA = csm, *sB = csm + CT * CLD, *sP = csm + 2 * CT * CLD;
  const int G = gridDim.x;
  GridBarrier bar(T.bar, (unsigned)G + T.bar_extra, T.err, T.bar_ns);
  GridBarrier sub(T.bar + 1, (unsigned)G, T.err, T.bar_ns);
  const bool lead = blockIdx.x == 0, solo = G == 1;
  const int me = solo ? 0 : (int)blockIdx.x - 1, others = solo ? 1 : G - 1;
  // tile 0's diagonal block
  if (lead) {
    load_potrf_tile(tile_at(T, 0, 0), sA);
    potrf_tile(tile_at(T, 0, 0), T.Linv, T.err, sA, sB, sP);
  }
  if (!bar.sync()) return;
  // With the inverse, X = L^-1 is formed in the same loop: tile row J of X
  // in phase T of column J (X_Jj = Linv_J R_Jj, its R final after the
  // updates of the earlier columns), and its updates R_Kj -= L_KJ X_Jj in
  // phase U -- the same products in the same order as a separate pass over
  // the tile rows, without its barriers.
  const int nxj = T.want_inverse ? 1 : 0;
  for (int J = 0; J < T.nt; ++J) {
    const int h = T.hrow[J], m = h - J;
    const int own = m > 0 ? 1 : 0;  // item 0 of T and of U is CTA 0's
    // T: L_IJ = A_IJ L_JJ^-T (items 0 .. m - 1); X_Jj = Linv_J R_Jj (items
    // m .. m + J with the inverse)
    if (lead && own) {
      __syncthreads();
      load_tile(sA, tile_at(T, J + 1, J), false);
      load_tile(sB, T.Linv + (size_t)J * TS, false);
      __syncthreads();
      double acc[NF][2] = {};
      gemm_nt(sA, sB, acc);
      store_frag(tile_at(T, J + 1, J), acc);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < NF; ++j)
        *(double2 *)(sA + frag_row() * CLD + frag_col() + 8 * j) = make_double2(acc[j][0], acc[j][1]);
    }
    const int ntt = m + nxj * (J + 1);
    if (!lead || solo)
      for (int t = own + me; t < ntt; t += others) {
        __syncthreads();
        double *gt;
        if (t < m) {
          gt = tile_at(T, J + 1 + t, J);
          load_tile(sA, gt, false);
          load_tile(sB, T.Linv + (size_t)J * TS, false);
        } else {
          gt = T.X + tri(J, t - m) * TS;
          load_tile(sA, T.Linv + (size_t)J * TS, false);
          load_tile(sB, gt, true);  // R^T: the product Linv R as Linv (R^T)^T
        }
        __syncthreads();
        double acc[NF][2] = {};
        gemm_nt(sA, sB, acc);
        __syncthreads();
        store_frag(gt, acc);
      }
    // U: A_IK -= L_IJ L_KJ^T (items 0 .. nu - 1).  With the inverse also
    // R_Kj -= L_KJ X_Jj, K > J, j <= J (items nu .. nu + m (J + 1) - 1).
    if (!lead || solo) {
      if (!sub.sync()) return;
      const long long nu = (long long)m * (m + 1) / 2;
      const long long ntu = nu + (long long)nxj * m * (J + 1);
      for (long long t = own + me; t < ntu; t += others) {
        __syncthreads();
        double *gt;
        if (t < nu) {
          int bi, bk;
          tri_item(t, bi, bk);
          load_tile(sA, tile_at(T, J + 1 + bi, J), false);
          load_tile(sB, tile_at(T, J + 1 + bk, J), false);
          gt = tile_at(T, J + 1 + bi, J + 1 + bk);
        } else {
          const long long u = t - nu;
          const int K = J + 1 + (int)(u / (J + 1)), j = (int)(u % (J + 1));
          load_tile(sA, tile_at(T, K, J), false);
          load_tile(sB, T.X + tri(J, j) * TS, true);
          gt = T.X + tri(K, j) * TS;
        }
        __syncthreads();
        double acc[NF][2] = {};
        gemm_nt(sA, sB, acc);
        sub_frag(gt, acc);
      }
    } else {
      sub.arrive();
    }
    if (lead && J + 1 < T.nt) {
      // the next diagonal tile: its last update from the tile of T in sA
      double *gt = tile_at(T, J + 1, J + 1);
      __syncthreads();
      if (own) {
        if (solo) {
          load_tile(sA, tile_at(T, J + 1, J), false);
          __syncthreads();
        }
        double acc[NF][2] = {};
        gemm_nt(sA, sA, acc);
        __syncthreads();
        sub_frag_to(gt, acc, sA);
      } else {
        load_potrf_tile(gt, sA);
      }
      potrf_tile(gt, T.Linv + (size_t)(J + 1) * TS, T.err, sA, sB, sP);
    }
    if (!bar.sync()) return;
  }
  if (!T.want_inverse) return;
  const int nt = T.nt;
  // A^-1 tile (i, k), k <= i: sum over m >= i of X_mi^T X_mk
  const long long no = (long long)nt * (nt + 1) / 2;
  for (long long t = blockIdx.x; t < no; t += G) {
    int bi, bk;
    tri_item(t, bi, bk);
    double acc[NF][2] = {};
    for (int mt = bi; mt < nt; ++mt) {
      __syncthreads();
      load_tile(sA, T.X + tri(mt, bi) * TS, true);
      load_tile(sB, T.X + tri(mt, bk) * TS, true);
      __syncthreads();
      gemm_nt(sA, sB, acc);
    }
    store_frag(T.Ainv + tri(bi, bk) * TS, acc);
  }
}

// Dense n x n row-major (lower triangle used), scaled by d_i d_j (+ eps on
// the diagonal), into lower tiles; the padding of the last diagonal tile is
// the identity.  X starts as the identity (diagonal tiles), zero elsewhere.
__global__ void k_pack_dense(const double *A, const double *dsc, double eps, int n, int nt, double *Lt, double *X) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ntile = (long long)nt * (nt + 1) / 2;
  if (idx >= ntile * TS) return;
  const long long t = idx / TS;
  const int e = (int)(idx % TS), a = e >> 6, b = e & 63;
  int I, J;
  tri_item(t, I, J);
  const int i = I * CT + a, j = J * CT + b;
  double v = 0.;
  if (i < n && j < n) {
    if (j <= i) {
      v = A[(size_t)i * n + j] * dsc[i] * dsc[j];
      if (i == j) v += eps;
    }
  } else if (i == j) {
    v = 1.;
  }
  Lt[idx] = v;
  X[idx] = (i == j) ? 1. : 0.;
}

// Lower inverse tiles back to the dense matrix (both triangles), scaled.
__global__ void k_unpack_dense(const double *At, const double *dsc, int n, int nt, double *Ainv) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ntile = (long long)nt * (nt + 1) / 2;
  if (idx >= ntile * TS) return;
  const long long t = idx / TS;
  const int e = (int)(idx % TS), a = e >> 6, b = e & 63;
  int I, J;
  tri_item(t, I, J);
  const int i = I * CT + a, j = J * CT + b;
  if (i >= n || j >= n || (I == J && b > a)) return;
  const double v = At[idx] * dsc[i] * dsc[j];
  Ainv[(size_t)i * n + j] = v;
  Ainv[(size_t)j * n + i] = v;
}

__global__ void k_dense_meta(int nt, long long *toff, int *fcol, int *hrow) {
  const int I = blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= nt) return;
  toff[I] = (long long)I * (I + 1) / 2;
  fcol[I] = 0;
  hrow[I] = nt - 1;
}

// one CTA per SM (fewer arrivals per grid barrier); 0 if none fits
int chol_grid() {
  int dev = 0, nsm = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(k_chol_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CSMEM);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_chol_tiles, CTH, CSMEM);
  return per >= 1 ? nsm : 0;
}

}  // namespace

// Factor the envelope tiles in place (L over A) and write the inverses of
// the diagonal tiles; one cooperative launch.  bar_extra, bar_ns: test hook
// (0, 0: none, the default limit).
void tile_cholesky(double *tiles, const long long *toff, const int *fcol, const int *hrow, double *Linv, int nt,
                   unsigned *bar, int *err, cudaStream_t s, unsigned bar_extra, unsigned long long bar_ns) {
  if (nt <= 0) return;
  Tiles T;
  T.L = tiles;
  T.toff = toff;
  T.fcol = fcol;
  T.hrow = hrow;
  T.Linv = Linv;
  T.X = nullptr;
  T.Ainv = nullptr;
  T.nt = nt;
  T.want_inverse = 0;
  T.bar = bar;
  T.err = err;
  T.bar_extra = bar_extra;
  T.bar_ns = bar_ns ? bar_ns : BAR_TIMEOUT_NS;
  const int g = std::max(1, chol_grid());
  RPBA_CUDA_CHECK(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s));
  void *args[] = {&T};
  RPBA_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)k_chol_tiles, dim3(g), dim3(CTH), args, CSMEM, s));
}

size_t spd_inverse_bytes(int n) {
  const long long nt = (n + CT - 1) / CT;
  return (size_t)(3 * (nt * (nt + 1) / 2) + nt) * TS * sizeof(double) + nt * 16 + 64;
}

// A^-1 of the dense SPD matrix (D A D + eps I) scaled back by D, with D =
// diag(dsc): A (row major n x n, lower triangle used) -> Ainv (both
// triangles).  One cooperative launch for the factorisation and the inverse.
void spd_inverse_scaled(const double *A, const double *dsc, double eps, int n, double *Ainv, void *work,
                        unsigned *bar, int *err, cudaStream_t s) {
  if (n <= 0) return;
  const int nt = (n + CT - 1) / CT;
  const long long ntile = (long long)nt * (nt + 1) / 2;
  double *Lt = (double *)work;
  double *X = Lt + ntile * TS;
  double *At = X + ntile * TS;
  double *Linv = At + ntile * TS;
  long long *toff = (long long *)(Linv + (size_t)nt * TS);
  int *fcol = (int *)(toff + nt);
  int *hrow = fcol + nt;
  k_dense_meta<<<(nt + 127) / 128, 128, 0, s>>>(nt, toff, fcol, hrow);
  k_pack_dense<<<(int)((ntile * TS + 255) / 256), 256, 0, s>>>(A, dsc, eps, n, nt, Lt, X);
  Tiles T;
  T.L = Lt;
  T.toff = toff;
  T.fcol = fcol;
  T.hrow = hrow;
  T.Linv = Linv;
  T.X = X;
  T.Ainv = At;
  T.nt = nt;
  T.want_inverse = 1;
  T.bar = bar;
  T.err = err;
  T.bar_extra = 0;
  T.bar_ns = BAR_TIMEOUT_NS;
  const int g = (int)std::max<long long>(1, std::min<long long>(chol_grid(), ntile));
  RPBA_CUDA_CHECK(cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s));
  void *args[] = {&T};
  RPBA_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)k_chol_tiles, dim3(g), dim3(CTH), args, CSMEM, s));
  k_unpack_dense<<<(int)((ntile * TS + 255) / 256), 256, 0, s>>>(At, dsc, n, nt, Ainv);
  RPBA_CUDA_CHECK(cudaGetLastError());
}

}  // namespace rpba
