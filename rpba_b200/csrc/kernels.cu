// kernels.cu -- per-observation, per-point and per-camera kernels of the
// global LSA (rbacore.cpp).  The linearisation kernels (point, camera,
// pair, back-substitution) are compiled for two forms: FP64 throughout (the
// drop-in form) and the mixed-precision form: FP32 records and blocks with
// FP32 arithmetic and compensated (Kahan) per-camera and per-pair sums, the
// point blocks factored in FP64 and the records whitened by the factor
// (k_point<float>).  Residuals and the cost stay FP64.
#include <cub/cub.cuh>

#include "internal.h"

namespace rpba {

namespace {

constexpr int GRP = 8;  // lanes per point in the point-major kernels

template <class T>
__device__ __forceinline__ T grp_sum(T v) {
#pragma unroll
  for (int o = GRP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, GRP);
  return v;
}

// Storage of the linearisation in either form.
template <class T>
struct Store;
template <>
struct Store<double> {
  static __device__ __forceinline__ double *rec(const DevLSA &L) { return L.rec; }
  static __device__ __forceinline__ double *ptV(const DevLSA &L) { return L.ptV; }
  static __device__ __forceinline__ double *blocks(const DevLSA &L) { return L.blocks; }
  static constexpr int BS = BS64;
};
template <>
struct Store<float> {
  static __device__ __forceinline__ float *rec(const DevLSA &L) { return L.rec32; }
  static __device__ __forceinline__ float *ptV(const DevLSA &L) { return L.ptV32; }
  static __device__ __forceinline__ float *blocks(const DevLSA &L) { return L.blocks32; }
  static constexpr int BS = BS32;
};

template <class T>
struct Pair2;
template <>
struct Pair2<float> {
  using type = float2;
};
template <>
struct Pair2<double> {
  using type = double2;
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Compensated (Kahan) accumulation for the FP32 form; plain in FP64.
template <class T>
struct Acc {
  T s = T(0), c = T(0);
  __device__ __forceinline__ void add(T x) {
    if constexpr (sizeof(T) == 4) {
      const T y = x - c;
      const T t = s + y;
      c = (t - s) - y;
      s = t;
    } else {
      s += x;
    }
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// In GCP mode camera 0 is free like the others and there is no scale
// camera (normcamera = -1; rbacore.cpp:697-698, 1005-1008).
__device__ __forceinline__ int role_of(const DevLSA &L, int k) {
  return (k == 0 && !L.ao) ? ROLE_ZERO : (k == L.normcamera ? ROLE_NORM : ROLE_FREE);
}

// ----------------------------------------------------------- cost pass
// CalcCorrections with derivflag = false (rbacore.cpp:1215-1331): per
// observation float cost term and the reweighting statistic sig0rmv.
__global__ void k_cost(DevLSA L, const double *__restrict__ XM, int srmv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.nobs) return;
  const int k = L.o_cam[i], p = L.o_pt[i];
  const double *X = XM + L.nrioff + 3 * p;
  const float2 xg = L.o_xg[i];
  ObsEval e;
  eval_obs(L.camn[k], X[0], X[1], X[2], xg.x, xg.y, L.defdiff, e);
  if (e.nan) {
    L.o_cost[i] = 0.f;
    L.o_s0rmv[i] = 1.e20f;
    return;
  }
  const float4 w = L.o_w[i];
  const float val = cost_term(e.d1, e.d2, w.x, w.y, w.z);
  L.o_cost[i] = val;
  if (srmv) {
    if (L.robust) {
      const float4 wo = L.o_wold[i];
      L.o_s0rmv[i] = cost_term(e.d1, e.d2, wo.x, wo.y, wo.z);
    } else {
      L.o_s0rmv[i] = val;
    }
  }
}

// GCP mode: the prior cost term of every point at the state XM, in the
// reference's float accumulation (sig0ao, rbacore.cpp:1677-1729): the double
// form d^T W d (d = gcp - X) in the reference's operation order, rounded to
// float; 0 for a point without a prior.
__global__ void k_gcp_cost(DevLSA L, const double *__restrict__ XM, float *out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= L.npts) return;
  float t = 0.f;
  const int gi = L.pt_gcp[p];
  if (gi > -1) {
    const float *w = L.W3 + 6 * (size_t)L.pt_w3row[p];
    const double *gx = L.gcpdata + 3 * (size_t)gi;
    const double *X = XM + L.nrioff + 3 * (size_t)p;
    const double d1 = __dsub_rn(gx[0], X[0]), d2 = __dsub_rn(gx[1], X[1]), d3 = __dsub_rn(gx[2], X[2]);
    const double a = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(d1, d1), (double)w[0]),
                                         __dmul_rn(__dmul_rn(d2, d2), (double)w[1])),
                               __dmul_rn(__dmul_rn(d3, d3), (double)w[2]));
    const double b = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(d1, d2), (double)w[3]),
                                         __dmul_rn(__dmul_rn(d1, d3), (double)w[4])),
                               __dmul_rn(__dmul_rn(d2, d3), (double)w[5]));
    t = __double2float_rn(__dadd_rn(a, __dmul_rn(2., b)));
  }
  out[p] = t;
}

// Sequential float sum in array order, terms of either sign: the reference
// accumulates its prior costs in float, one point after the other
// (rbacore.cpp:1677-1729).  Warp 0 runs the chain of additions on values the
// other warps stage in shared memory a block ahead (16-byte broadcast loads,
// so the chain is the additions alone); with the values passed by shuffle a
// term took 25 cycles.
constexpr int SS_T = 256, SS_B = 2048;
__global__ void __launch_bounds__(SS_T) k_seq_sum(const float *__restrict__ v, int n, float *out) {
  __shared__ __align__(16) float buf[2][SS_B];
  const int tid = threadIdx.x;
  for (int j = tid; j < SS_B; j += SS_T)
    if (j < n) buf[0][j] = v[j];
  __syncthreads();
  float s = 0.f;
  for (int base = 0, b = 0; base < n; base += SS_B, b ^= 1) {
    if (tid < 32) {
      const int cnt = min(SS_B, n - base);
      int j = 0;
#pragma unroll 4
      for (; j + 4 <= cnt; j += 4) {
        const float4 a = *(const float4 *)(buf[b] + j);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
      }
      for (; j < cnt; ++j) s = __fadd_rn(s, buf[b][j]);
    } else {
      for (int j = tid - 32; j < SS_B; j += SS_T - 32)
        if (base + SS_B + j < n) buf[b ^ 1][j] = v[base + SS_B + j];
    }
    __syncthreads();
  }
  if (tid == 0) *out = s;
}

// ---------------------------------------------------------- point pass
// CalcCorrections/CalcDerivatives with derivflag = true, solveflag = false
// (rbacore.cpp:1215-1348, 1420-1616): Jacobians of every observation, the
// point block V = sum Jp^T W Jp and g = sum Jp^T W d, V damped and inverted;
// the per-observation record for the camera, pair and back-substitution
// kernels.
//
// FP32 form: whitened.  V and g are summed in FP64 from
// the FP32-rounded point Jacobians, V = L L^T is factored in FP64, and the
// record carries H = G L^-T in place of G, so that every Schur product
// G V^-1 G^T = H H^T is formed from bounded factors (H H^T <= W for each
// observation) however ill-conditioned V is: the explicit V^-1 of a distant,
// down-weighted point overflows FP32, and products with it lose all digits.
// A pivot at or below 1e-13 of its diagonal entry (not resolvable in FP64
// arithmetic) or below 1e-60 drops its coordinate: the step leaves that
// coordinate of the point unchanged (the factor is that of V without its row
// and column), and the Schur contribution stays positive semidefinite.
// Point record: L^-1 (9, row major, zeros above the diagonal), q = L^-1 g.
//
// A warp takes PT_N consecutive points, whose observations are consecutive
// too, 32 at a time whichever point they belong to.  Every lane leaves its
// observation's record and its terms of V and g in shared memory; four lanes
// a point then sum the terms (eight running sums a point, observations l,
// l + 8, ... in sum l, then a butterfly) and factor V, and the records are
// finished and written out 16 bytes a lane along the lines.  Observations
// before the last 32 wait in global memory.  Bound by the latency of the
// camera states and of the FP64 divisions and roots at 12 to 16 warps an SM:
// eight lanes a point, in turns of eight observations, ran 1.9 turns for
// every four points of a city (the longest of the four decides), each lane
// writing its own record, 32 lines an instruction.  A launch: FP32, 27.8M
// observations 3.95 -> 2.8 ms, 868,000 155 -> 97 us; FP64, 2.8M 0.58 -> 0.42
// ms, 902,000 191 -> 141 us.
template <class T>
struct PointGeom {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int RS = REC + 16 / (int)sizeof(T);  // values per record in shared memory (odd number of pieces)
  static constexpr int NC = F32 ? 9 : 12, CS = F32 ? 9 : 13;  // terms of V and g, stride
  static constexpr int NM = F32 ? 9 : 12;                     // per point: factor and q, or V^-1 and V^-1 g
  static constexpr int W = F32 ? 4 : 2;                       // warps per CTA (48 KB of shared memory at most)
};
constexpr int PT_N = 8;  // points per warp
template <class T>
struct PointShared {
  using Ge = PointGeom<T>;
  T rec[32 * Ge::RS];
  double term[32 * Ge::CS], acc[2 * Ge::NC][32], pt[PT_N][Ge::NM];
};

template <class T>
__global__ void __launch_bounds__(32 * PointGeom<T>::W, sizeof(T) == 4 ? 4 : 6) k_point(DevLSA L, double multfact1) {
  using Ge = PointGeom<T>;
  constexpr bool F32 = Ge::F32;
  constexpr int RS = Ge::RS, NC = Ge::NC, CS = Ge::CS;
  constexpr int PR = REC * (int)sizeof(T) / 16;  // pieces of a record
  extern __shared__ __align__(16) unsigned char pt_dyn[];
  PointShared<T> &S = ((PointShared<T> *)pt_dyn)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, p0 = (blockIdx.x * Ge::W + (threadIdx.x >> 5)) * PT_N;
  if (p0 >= L.npts) return;
  const int pn = min(PT_N, L.npts - p0);
  T *rec = Store<T>::rec(L);
  // the lane's point (four lanes each) and the warp's observations
  const int q = lane >> 2, j = lane & 3;
  const int base = L.pt_off[p0], end = L.pt_off[p0 + pn];
  const int t0 = q < pn ? L.pt_off[p0 + q] : end, t1 = q < pn ? L.pt_off[p0 + q + 1] : end;
  const int esvm[2] = {L.gauge[0], L.gauge[1]};
  T *r = S.rec + lane * RS;
  // records of the observations wb .. wb + 31: shared memory to global and back
  auto copy_out = [&](int wb) {
    __syncwarp();
    const int n = min(32, end - wb) * PR;
    float4 *dst = (float4 *)(rec + (size_t)wb * REC);
#pragma unroll
    for (int it = 0; it < PR; ++it) {
      const int i = lane + 32 * it;
      if (i < n) dst[i] = *(const float4 *)(S.rec + (i / PR) * RS + (i % PR) * (16 / (int)sizeof(T)));
    }
    __syncwarp();
  };
  auto copy_in = [&](int wb) {
    const float4 *src = (const float4 *)(rec + (size_t)wb * REC);
#pragma unroll
    for (int it = 0; it < PR; ++it) {
      const int i = lane + 32 * it;  // (only the last 32 can be fewer, and they never left)
      *(float4 *)(S.rec + (i / PR) * RS + (i % PR) * (16 / (int)sizeof(T))) = src[i];
    }
    __syncwarp();
  };
  double va[NC], vb[NC];  // running sums j and j + 4 of the point
  for (int wb = base; wb < end || wb == base; wb += 32) {
    const int o = wb + lane;
    if (o < end) {
      const int k = L.o_cam[o];
      const double *X = L.XPM + L.nrioff + 3 * (size_t)L.o_pt[o];
      const CamState c = L.camn[k];
      const float2 xg = L.o_xg[o];
      ObsEval e;
      eval_obs(c, X[0], X[1], X[2], xg.x, xg.y, L.defdiff, e);
      if (e.nan) L.o_s0rmv[o] = 1.e20f;
      T Bc[2][RPBA_P], Bp[2][3];
      jacobians<T>(c, e, role_of(L, k), esvm, L.addmask, Bc, Bp);
      const bool cam_active = k >= L.begini;
#pragma unroll
      for (int h = 0; h < RPBA_P; ++h) {
        typename Pair2<T>::type v;
        v.x = cam_active ? Bc[0][h] : T(0);
        v.y = cam_active ? Bc[1][h] : T(0);
        *(typename Pair2<T>::type *)(r + 2 * h) = v;
      }
      const float4 w = L.o_w[o];
      const double W0 = w.x, W1 = w.y, W2 = w.z;
      double *t = S.term + lane * CS;
      double G[2][3];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        G[0][h] = Bp[0][h] * W0 + Bp[1][h] * W2;
        G[1][h] = Bp[0][h] * W2 + Bp[1][h] * W1;
      }
      if constexpr (F32) {
        t[0] = G[0][0] * Bp[0][0] + G[1][0] * Bp[1][0];
        t[1] = G[0][0] * Bp[0][1] + G[1][0] * Bp[1][1];
        t[2] = G[0][0] * Bp[0][2] + G[1][0] * Bp[1][2];
        t[3] = G[0][1] * Bp[0][1] + G[1][1] * Bp[1][1];
        t[4] = G[0][1] * Bp[0][2] + G[1][1] * Bp[1][2];
        t[5] = G[0][2] * Bp[0][2] + G[1][2] * Bp[1][2];
#pragma unroll
        for (int a = 0; a < 3; ++a) t[6 + a] = G[0][a] * e.d1 + G[1][a] * e.d2;
        // Jp until the factor is known (then H)
#pragma unroll
        for (int h = 0; h < 3; ++h) {
          r[18 + h] = Bp[0][h];
          r[21 + h] = Bp[1][h];
        }
      } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
          for (int b = 0; b < 3; ++b) t[a * 3 + b] = G[0][a] * Bp[0][b] + G[1][a] * Bp[1][b];
          t[9 + a] = G[0][a] * e.d1 + G[1][a] * e.d2;
        }
#pragma unroll
        for (int h = 0; h < 3; ++h) {
          r[18 + h] = G[0][h];
          r[21 + h] = G[1][h];
        }
      }
      r[24] = (T)(e.d1 * W0 + e.d2 * W2);
      r[25] = (T)(e.d1 * W2 + e.d2 * W1);
    }
    __syncwarp();
#pragma unroll
    for (int f = 0; f < NC; ++f) {
      va[f] = wb > base ? S.acc[f][lane] : 0.;
      vb[f] = wb > base ? S.acc[NC + f][lane] : 0.;
    }
    int u = t0 + j;
    if (u < wb) u += ((wb - u) >> 3) << 3;
    const int ue = min(t1, wb + 32);
    for (; u < ue; u += 8) {
      if (u >= wb) {
        const double *t = S.term + (u - wb) * CS;
#pragma unroll
        for (int f = 0; f < NC; ++f) va[f] += t[f];
      }
      if (u + 4 >= wb && u + 4 < ue) {
        const double *t = S.term + (u + 4 - wb) * CS;
#pragma unroll
        for (int f = 0; f < NC; ++f) vb[f] += t[f];
      }
    }
    if (wb + 32 < end) {
#pragma unroll
      for (int f = 0; f < NC; ++f) {
        S.acc[f][lane] = va[f];
        S.acc[NC + f][lane] = vb[f];
      }
      copy_out(wb);
    }
  }
#pragma unroll
  for (int f = 0; f < NC; ++f) {
    va[f] += vb[f];
    va[f] += __shfl_xor_sync(0xffffffffu, va[f], 2);
    va[f] += __shfl_xor_sync(0xffffffffu, va[f], 1);
  }
  const int p = p0 + q;
  T *pv = Store<T>::ptV(L) + (size_t)p * PREC;
  if constexpr (F32) {
    double V[6], g[3];
#pragma unroll
    for (int f = 0; f < 6; ++f) V[f] = va[f];
#pragma unroll
    for (int f = 0; f < 3; ++f) g[f] = va[6 + f];
    V[0] *= multfact1;
    V[3] *= multfact1;
    V[5] *= multfact1;
    // V = L L^T with guarded pivots; m = L^-1 (lower)
    auto root = [](double d, double diag) { return (d > 1.e-13 * diag && d > 1.e-60) ? sqrt(d) : 0.; };
    const double l00 = root(V[0], V[0]);
    const double i00 = l00 > 0. ? 1. / l00 : 0.;
    const double l10 = V[1] * i00, l20 = V[2] * i00;
    const double l11 = root(V[3] - l10 * l10, V[3]);
    const double i11 = l11 > 0. ? 1. / l11 : 0.;
    const double l21 = (V[4] - l20 * l10) * i11;
    const double l22 = root(V[5] - l20 * l20 - l21 * l21, V[5]);
    const double i22 = l22 > 0. ? 1. / l22 : 0.;
    double m[6] = {i00, -l10 * i00 * i11, i11, -(l20 * i00 - l21 * l10 * i00 * i11) * i22, -l21 * i11 * i22, i22};
    // m00 m10 m11 m20 m21 m22; a factor beyond the FP32 range drops the point
    bool inrange = true;
#pragma unroll
    for (int f = 0; f < 6; ++f) inrange = inrange && fabs(m[f]) < 1.e30;
    if (!inrange)
#pragma unroll
      for (int f = 0; f < 6; ++f) m[f] = 0.;
    const double q0 = m[0] * g[0], q1 = m[1] * g[0] + m[2] * g[1], q2 = m[3] * g[0] + m[4] * g[1] + m[5] * g[2];
    if (j == 0 && q < pn) {
#pragma unroll
      for (int f = 0; f < 6; ++f) S.pt[q][f] = m[f];
      S.pt[q][6] = q0;
      S.pt[q][7] = q1;
      S.pt[q][8] = q2;
      ((float4 *)pv)[0] = make_float4((float)m[0], 0.f, 0.f, (float)m[1]);
      ((float4 *)pv)[1] = make_float4((float)m[2], 0.f, (float)m[3], (float)m[4]);
      ((float4 *)pv)[2] = make_float4((float)m[5], (float)q0, (float)q1, (float)q2);
    }
  } else {
    double V[9], g[3];
#pragma unroll
    for (int f = 0; f < 9; ++f) V[f] = va[f];
#pragma unroll
    for (int f = 0; f < 3; ++f) g[f] = va[9 + f];
    if (L.ao && q < pn && L.pt_gcp[p] > -1) {
      // CalcDerivatives3DGCP (rbacore.cpp:1677-1729): the 3-D prior of a
      // point shared with other partitions, residual gcp - X, B = -I
      const double *X = L.XPM + L.nrioff + 3 * (size_t)p;
      const float *w = L.W3 + 6 * (size_t)L.pt_w3row[p];
      const double *gx = L.gcpdata + 3 * (size_t)L.pt_gcp[p];
      const double d1 = gx[0] - X[0], d2 = gx[1] - X[1], d3 = gx[2] - X[2];
      const double Wm[9] = {w[0], w[3], w[4], w[3], w[1], w[5], w[4], w[5], w[2]};
#pragma unroll
      for (int f = 0; f < 9; ++f) V[f] += Wm[f];
#pragma unroll
      for (int f = 0; f < 3; ++f) g[f] += (-Wm[f * 3]) * d1 + (-Wm[f * 3 + 1]) * d2 + (-Wm[f * 3 + 2]) * d3;
    }
    V[0] = V[0] * multfact1;
    V[4] = V[4] * multfact1;
    V[8] = V[8] * multfact1;
    double Vi[9];
    inv3<double>(V, Vi);
    if (j == 0 && q < pn) {
#pragma unroll
      for (int f = 0; f < 9; ++f) S.pt[q][f] = pv[f] = Vi[f];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        pv[9 + a] = g[a];
        S.pt[q][9 + a] = Vi[a * 3] * g[0] + Vi[a * 3 + 1] * g[1] + Vi[a * 3 + 2] * g[2];
      }
    }
  }
  __syncwarp();
  // the last 32 observations' records are in shared memory, the others return
  bool here = true;
  for (int wb = base + ((max(end - base, 1) - 1) / 32) * 32; wb >= base; wb -= 32) {
    if (!here) copy_in(wb);
    here = false;
    const int o = wb + lane;
    if (o < end) {
      const double *m = S.pt[L.o_pt[o] - p0];
      const float4 w = L.o_w[o];
      if constexpr (F32) {
        const double W0 = w.x, W1 = w.y, W2 = w.z;
        const float4 ra = *(const float4 *)(r + 16), rb = *(const float4 *)(r + 20);
        const float2 e = *(const float2 *)(r + 24);
        double H[2][3];
        {
          const double p00 = ra.z, p01 = ra.w, p02 = rb.x, p10 = rb.y, p11 = rb.z, p12 = rb.w;
          const double G0[3] = {p00 * W0 + p10 * W2, p01 * W0 + p11 * W2, p02 * W0 + p12 * W2};
          const double G1[3] = {p00 * W2 + p10 * W1, p01 * W2 + p11 * W1, p02 * W2 + p12 * W1};
          H[0][0] = m[0] * G0[0];
          H[0][1] = m[1] * G0[0] + m[2] * G0[1];
          H[0][2] = m[3] * G0[0] + m[4] * G0[1] + m[5] * G0[2];
          H[1][0] = m[0] * G1[0];
          H[1][1] = m[1] * G1[0] + m[2] * G1[1];
          H[1][2] = m[3] * G1[0] + m[4] * G1[1] + m[5] * G1[2];
        }
        const double h00 = H[0][0] * H[0][0] + H[0][1] * H[0][1] + H[0][2] * H[0][2];
        const double h01 = H[0][0] * H[1][0] + H[0][1] * H[1][1] + H[0][2] * H[1][2];
        const double h11 = H[1][0] * H[1][0] + H[1][1] * H[1][1] + H[1][2] * H[1][2];
        // H at 18..23, W - H H^T at 26..28, W d - H q at 29, 30, 31 zero
        float4 *r4 = (float4 *)(r + 16);
        r4[0] = make_float4(ra.x, ra.y, (float)H[0][0], (float)H[0][1]);
        r4[1] = make_float4((float)H[0][2], (float)H[1][0], (float)H[1][1], (float)H[1][2]);
        r4[2] = make_float4(e.x, e.y, (float)(W0 - h00), (float)(W2 - h01));
        r4[3] = make_float4((float)(W1 - h11), (float)((double)e.x - (H[0][0] * m[6] + H[0][1] * m[7] + H[0][2] * m[8])),
                            (float)((double)e.y - (H[1][0] * m[6] + H[1][1] * m[7] + H[1][2] * m[8])), 0.f);
      } else {
        double G[2][3], GV[2][3];
#pragma unroll
        for (int h = 0; h < 3; ++h) {
          G[0][h] = r[18 + h];
          G[1][h] = r[21 + h];
        }
        const double *vg = m + 9;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) GV[a][b] = G[a][0] * m[b] + G[a][1] * m[3 + b] + G[a][2] * m[6 + b];
        r[26] = (T)w.x - (GV[0][0] * G[0][0] + GV[0][1] * G[0][1] + GV[0][2] * G[0][2]);
        r[27] = (T)w.z - (GV[0][0] * G[1][0] + GV[0][1] * G[1][1] + GV[0][2] * G[1][2]);
        r[28] = (T)w.y - (GV[1][0] * G[1][0] + GV[1][1] * G[1][1] + GV[1][2] * G[1][2]);
        r[29] = r[24] - (G[0][0] * vg[0] + G[0][1] * vg[1] + G[0][2] * vg[2]);
        r[30] = r[25] - (G[1][0] * vg[0] + G[1][1] * vg[1] + G[1][2] * vg[2]);
        r[31] = 0.;
      }
    }
    copy_out(wb);
  }
}

// --------------------------------------------------------- camera pass
// Diagonal blocks of the reduced camera system and its right-hand side:
// S_kk = sum_o Bc^T (W - G V^-1 G^T) Bc, b_k = sum_o Bc^T (W d - G V^-1 g)
// (the camera terms of rbacore.cpp:1552-1561 minus the Schur terms of
// :1358-1360), then the damping of rbacore.cpp:1164-1170.  A CTA per camera:
// three warps bring its observations in the reference's nro order, chunk by
// chunk -- eight observations a warp by asynchronous copies two chunks ahead,
// then, one chunk ahead, T = (M Bc, m) by four lanes an observation -- and
// the first warp's lanes add every observation to two entries (i, j),
// (i, j + 1) of the upper triangle or the right-hand side (column 9) each.
// Few cameras leave it to the latency of the adding warp, many to the bytes
// shared memory hands to registers; two warps that each staged, transformed
// and added in turn took 47 us for 12 cameras of 470 observations (now 22),
// 0.41 ms for 1,000 of 900 (0.17), FP32 2.3 ms for 13,700 of 2,000 (0.95; a
// warp a camera that does all three in turn 0.92, but 35 us and 0.29 ms).
constexpr int CAM_W = 4, CAM_O = 8, CAM_B = (CAM_W - 1) * CAM_O;  // warps; observations per warp, per chunk
template <class T>
struct CamGeom {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int V16 = 16 / sizeof(T);                 // values per 16-byte piece
  static constexpr int P0 = F32 ? 5 : 9, P1 = F32 ? 2 : 3;   // pieces: Bc; M and m
  static constexpr int R1 = F32 ? 24 : 26, O1 = P0 * V16;    // M's pieces in the record and in the stage
  static constexpr int OM = O1 + 26 - R1;                    // M00, M01, M11, m0, m1
  static constexpr int OT = (P0 + P1) * V16;                 // T, ten pairs
  static constexpr int ST = F32 ? 52 : 46;                   // an odd number of pieces (bank conflicts)
};

template <class T>
__global__ void __launch_bounds__(32 * CAM_W, 6) k_camera(DevLSA L, double multfact1) {
  using Ge = CamGeom<T>;
  using V2 = typename Pair2<T>::type;
  constexpr int ST = Ge::ST, PC = Ge::P0 + Ge::P1, V16 = Ge::V16;
  const int k = blockIdx.x + L.begini, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (k >= L.nimg) return;
  __shared__ __align__(16) T stage[3][CAM_B * ST];
  const int beg = L.coff[k], end = L.coff[k + 1], nchunk = (end - beg + CAM_B - 1) / CAM_B;
  if (warp > 0) {
    const T *rec = Store<T>::rec(L);
    const int w0 = (warp - 1) * CAM_O;  // the warp's observations of a chunk
    auto idx_of = [&](int c) {
      const int t = beg + c * CAM_B + w0 + lane;
      return lane < CAM_O && t < end ? __ldg(L.camlist + t) : 0;
    };
    auto issue = [&](int c, int ol) {
      const int n = min(CAM_O, end - (beg + c * CAM_B + w0));
      T *b = stage[c % 3] + w0 * ST;
#pragma unroll
      for (int m = 0; m < (CAM_O * PC + 31) / 32; ++m) {
        const int t = lane + 32 * m, ob = t / PC, e = t - ob * PC;
        const int o = __shfl_sync(0xffffffffu, ol, ob & 31);
        if (ob < n)
          cp_async16(b + ob * ST + e * V16,
                     rec + (size_t)o * REC + (e < Ge::P0 ? e * V16 : Ge::R1 + (e - Ge::P0) * V16));
      }
      cp_async_commit();
    };
    auto form = [&](int c) {
      const int ob = lane & 7, g = lane >> 3;
      if (beg + c * CAM_B + w0 + ob < end) {
        T *r = stage[c % 3] + (w0 + ob) * ST;
        const T M00 = r[Ge::OM], M01 = r[Ge::OM + 1], M11 = r[Ge::OM + 2];
#pragma unroll
        for (int h = 0; h < 3; ++h) {
          const int q = g + 4 * h;
          if (q > 9) continue;
          V2 t;
          if (q < 9) {
            const V2 v = *(const V2 *)(r + 2 * q);
            t.x = M00 * v.x + M01 * v.y;
            t.y = M01 * v.x + M11 * v.y;
          } else {
            t.x = r[Ge::OM + 3];
            t.y = r[Ge::OM + 4];
          }
          *(V2 *)(r + Ge::OT + 2 * q) = t;
        }
      }
    };
    // (a group a chunk, empty past the last one)
    issue(0, idx_of(0));
    int ol = idx_of(1);
    issue(1, ol);
    ol = idx_of(2);
    cp_async_wait<1>();
    __syncwarp();
    form(0);
    __syncthreads();
    for (int c = 0; c < nchunk; ++c) {
      issue(c + 2, ol);
      ol = idx_of(c + 3);
      cp_async_wait<1>();
      __syncwarp();
      form(c + 1);
      __syncthreads();
    }
    cp_async_wait<0>();
    return;
  }
  // the lane's entries (i, j) and (i, j + 1), j + 1 <= 9
  int i = 0, j = lane;
  while (i < 9 && j >= (11 - i) / 2) j -= (11 - i++) / 2;
  j = i + 2 * j;
  const bool v0 = i < 9, v1 = v0 && j + 1 <= 9;
  const int ic = v0 ? i : 0, j0 = v0 ? j : 0, j1 = v1 ? j + 1 : j0;
  Acc<T> acc0, acc1;
  __syncthreads();
  for (int c = 0; c < nchunk; ++c) {
    const int n = min(CAM_B, end - beg - c * CAM_B);
    const T *b = stage[c % 3], *pa = b + 2 * ic, *p0 = b + Ge::OT + 2 * j0, *p1 = b + Ge::OT + 2 * j1;
#pragma unroll 4
    for (int ob = 0; ob < n; ++ob) {
      const V2 a = *(const V2 *)(pa + ob * ST), c0 = *(const V2 *)(p0 + ob * ST), c1 = *(const V2 *)(p1 + ob * ST);
      acc0.add(a.x * c0.x + a.y * c0.y);
      acc1.add(a.x * c1.x + a.y * c1.y);
    }
    __syncthreads();
  }
  const int np = L.camparv[k + 1] - L.camparv[k];
  T *D = Store<T>::blocks(L) + (size_t)k * Store<T>::BS;
  auto put = [&](int jj, double v) {
    if (jj == 9) {
      L.rhs[k * 9 + i] = i < np ? (double)(T)v : 0.;
      return;
    }
    if (i < np && jj < np) {
      if (i == jj) v = __dadd_rn(__dmul_rn(v, multfact1), 1.e-2);
    } else {
      v = i == jj ? 1. : 0.;
    }
    D[i * 9 + jj] = (T)v;
    D[jj * 9 + i] = (T)v;
  };
  if (v0) put(j, acc0.value());
  if (v1) put(j + 1, acc1.value());
}

// ----------------------------------------------------------- pair pass
// Off-diagonal blocks: S_kl = - sum_p W_pk V_p^-1 W_pl^T over the points
// seen by both cameras (rbacore.cpp:1362-1390), with W_po = Bc^T G.  One
// warp per block sums its contributions in a fixed order (the FP32 form in
// chunks of 32, each added into a compensated sum).  Both forms take a chunk
// (PairGeom::CH) in three steps: the records by 16-byte asynchronous copies
// into shared memory; a lane (FP64: two) a contribution, the 2 x 2 product N
// of the points' part -- FP32 G V^-1 G^T = H H^T of the whitened records --
// and with it one side's Bc, in place; then lanes 0..26 add every
// contribution to three entries each, (i, 3 g .. 3 g + 2).
// What bounds it are instructions (FP64: the FP64 units) and the bytes that
// shared memory hands to registers (FP32: eight values a lane and
// contribution, 79% of the cycles), not HBM.  With N formed by every lane and
// the records staged through registers one contribution ahead the FP32 form
// took twice the instructions: 5.5M blocks, 28M observations 11.9 -> 8.9 ms
// a launch; FP64, 365,000 blocks 2.72 -> 1.50 ms, 33,000 blocks of a chain
// 1.09 -> 0.44 ms, 66 blocks (latency) 94 -> 33 us.  Two stages in flight were
// no faster but for the smallest (33 -> 29 us), fewer registers (7 or 8 CTAs
// an SM) slower by their spills in the FP64 form.
template <class T>
struct PairGeom {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int CH = F32 ? 32 : 16;     // contributions per stage
  static constexpr int V16 = 16 / sizeof(T);   // values per 16-byte piece
  static constexpr int PR = 24 / V16;          // pieces of a record's Bc and G (H)
  static constexpr int PP = F32 ? 0 : 5;       // and of the point's V^-1
  static constexpr int PC = 2 * PR + PP;
  // values per contribution: an odd number of 16-byte pieces, so that the
  // lanes of a quarter warp meet no bank twice
  static constexpr int ST = F32 ? 52 : 58;
  static constexpr int STAGE_BYTES = CH * (ST * (int)sizeof(T) + (F32 ? 8 : 16));
};
constexpr int PAIR_W = 4;  // warps per CTA

template <class T>
__global__ void __launch_bounds__(32 * PAIR_W, sizeof(T) == 4 ? 6 : 5) k_pair(DevLSA L) {
  using Ge = PairGeom<T>;
  constexpr bool F32 = Ge::F32;
  constexpr int CH = Ge::CH, ST = Ge::ST, PR = Ge::PR, PC = Ge::PC, V16 = Ge::V16;
  const int wid = blockIdx.x * PAIR_W + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (wid >= L.nboff) return;
  __shared__ __align__(16) unsigned char stages[PAIR_W * Ge::STAGE_BYTES];
  unsigned char *mine = stages + (size_t)(threadIdx.x >> 5) * Ge::STAGE_BYTES;
  const T *rec = Store<T>::rec(L), *ptv = Store<T>::ptV(L);
  const int cb = L.boff[wid], ce = L.boff[wid + 1];
  // the contributions of the chunk at c0, one per lane, and its points
  auto pair_of = [&](int c0) { return lane < CH && c0 + lane < ce ? __ldg(L.contrib + c0 + lane) : make_int2(0, 0); };
  auto point_of = [&](int2 pr, int c0) { return !F32 && lane < CH && c0 + lane < ce ? __ldg(L.o_pt + pr.x) : 0; };
  // copy the chunk's records to the stage
  auto issue = [&](int c0, int2 pr, int pp) {
    int *si = (int *)(mine + CH * ST * (int)sizeof(T));
    const int n = min(CH, ce - c0);
    if (lane < CH) {
      if constexpr (F32)
        ((int2 *)si)[lane] = pr;
      else
        ((int4 *)si)[lane] = make_int4(pr.x, pr.y, pp, 0);
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < (CH * PC + 31) / 32; ++m) {
      if (32 * m >= n * PC) break;
      const int t = lane + 32 * m;
      if (t < n * PC) {
        const int c = t / PC, e = t - c * PC, w = F32 || e < 2 * PR ? e / PR : 2, f = (e - w * PR) * V16;
        const int o = si[(F32 ? 2 : 4) * c + w];
        const T *src = w < 2 ? rec + (size_t)o * REC + f : ptv + (size_t)o * PREC + f;
        cp_async16((T *)mine + c * ST + 24 * w + f, src);
      }
    }
  };
  const int i = lane < 27 ? lane / 3 : 0, g = lane < 27 ? lane - 3 * (lane / 3) : 0;
  T ks[3] = {T(0), T(0), T(0)}, kc[3] = {T(0), T(0), T(0)};
  // contributions two chunks ahead, points one chunk ahead
  int2 pr1 = pair_of(cb), pr2 = pair_of(cb + CH);
  int pp1 = point_of(pr1, cb);
  issue(cb, pr1, pp1);
  pp1 = point_of(pr2, cb + CH);
  pr1 = pr2;
  pr2 = pair_of(cb + 2 * CH);
  T *b = (T *)mine;
  for (int c0 = cb; c0 < ce; c0 += CH) {
    const int n = min(CH, ce - c0);
    cp_async_wait_all();
    __syncwarp();
    if constexpr (F32) {
      // a lane a contribution: U = Bc_k^T N, N = H_k H_l^T, in place of Bc_k
      float *r = (float *)b + lane * ST;
      if (lane < n) {
        float x[24];
#pragma unroll
        for (int v = 0; v < 6; ++v) *(float4 *)(x + 4 * v) = *(const float4 *)(r + 4 * v);
        const float2 y0 = *(const float2 *)(r + 42);
        const float4 y1 = *(const float4 *)(r + 44);
        const float n00 = x[18] * y0.x + x[19] * y0.y + x[20] * y1.x;
        const float n01 = x[18] * y1.y + x[19] * y1.z + x[20] * y1.w;
        const float n10 = x[21] * y0.x + x[22] * y0.y + x[23] * y1.x;
        const float n11 = x[21] * y1.y + x[22] * y1.z + x[23] * y1.w;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          const float b0 = x[2 * k], b1 = x[2 * k + 1];
          x[2 * k] = b0 * n00 + b1 * n10;
          x[2 * k + 1] = b0 * n01 + b1 * n11;
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) *(float4 *)(r + 4 * v) = *(const float4 *)(x + 4 * v);
        *(float2 *)(r + 16) = make_float2(x[16], x[17]);
      }
    } else {
      // two lanes a contribution: T = N Bc_l, N = G_k V^-1 G_l^T, in place
      // of Bc_l (one lane columns 0 .. 4, the other the rest)
      double *r = (double *)b + (lane & 15) * ST;
      if ((lane & 15) < n) {
        double Gs[6], Gt[6], Vi[10];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          *(double2 *)(Gs + 2 * v) = *(const double2 *)(r + 18 + 2 * v);
          *(double2 *)(Gt + 2 * v) = *(const double2 *)(r + 42 + 2 * v);
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) *(double2 *)(Vi + 2 * v) = *(const double2 *)(r + 48 + 2 * v);
        double GV[2][3], N[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            GV[a][c] = Gs[a * 3] * Vi[c] + Gs[a * 3 + 1] * Vi[3 + c] + Gs[a * 3 + 2] * Vi[6 + c];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int c = 0; c < 2; ++c)
            N[a][c] = GV[a][0] * Gt[c * 3] + GV[a][1] * Gt[c * 3 + 1] + GV[a][2] * Gt[c * 3 + 2];
        const int k0 = lane < 16 ? 0 : 5;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          if (k0 + k < 9) {
            double2 *q = (double2 *)(r + 24 + 2 * (k0 + k));
            const double2 bt = *q;
            *q = make_double2(N[0][0] * bt.x + N[0][1] * bt.y, N[1][0] * bt.x + N[1][1] * bt.y);
          }
        }
      }
    }
    __syncwarp();
    // every lane its three entries (i, 3 g .. 3 g + 2), in the contributions' order
    T part[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) part[q] = F32 ? T(0) : ks[q];
    const T *pa = b + 2 * i, *pc = b + 24 + 6 * g;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
      const typename Pair2<T>::type a = *(const typename Pair2<T>::type *)(pa + j * ST);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const typename Pair2<T>::type c = *(const typename Pair2<T>::type *)(pc + j * ST + 2 * q);
        part[q] -= a.x * c.x + a.y * c.y;
      }
    }
    __syncwarp();
    if constexpr (F32) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const float y = part[q] - kc[q];
        const float t = ks[q] + y;
        kc[q] = (t - ks[q]) - y;
        ks[q] = t;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q) ks[q] = part[q];
    }
    if (c0 + CH < ce) issue(c0 + CH, pr1, pp1);
    pp1 = point_of(pr2, c0 + 2 * CH);
    pr1 = pr2;
    pr2 = pair_of(c0 + 3 * CH);
  }
  if (lane < 27) {
    T *B = Store<T>::blocks(L) + (size_t)(L.nimg + wid) * Store<T>::BS + i * 9 + 3 * g;
#pragma unroll
    for (int q = 0; q < 3; ++q) __stcs(B + q, F32 ? (T)((double)ks[q] - (double)kc[q]) : ks[q]);  // keep L2 for the records
  }
}

// ------------------------------------------------- back-substitution
// rbacore.cpp:1395-1410: dX_p = V^-1 (g - sum_o W_o^T dc_k), with
// W_o^T dc = G^T (Bc dc); in the FP32 form L^-T (q - sum_o H^T (Bc dc)).
template <class T>
__global__ void k_backsub(DevLSA L, const double *__restrict__ xsol) {
  const int gt = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = gt / GRP, ln = gt % GRP;
  const bool valid = p < L.npts;  // no early exit (full-warp shuffles below)
  const int t0 = valid ? L.pt_off[p] : 0, t1 = valid ? L.pt_off[p + 1] : 0;
  T a0 = 0., a1 = 0., a2 = 0.;
  for (int o = t0 + ln; o < t1; o += GRP) {
    const int k = L.o_cam[o];
    if (k < L.begini) continue;
    const T *rp = Store<T>::rec(L) + (size_t)o * REC;
    const double *dc = xsol + (size_t)k * 9;
    T r[24];
    if constexpr (sizeof(T) == 4) {
      // the FP32 record's first 24 floats in six 16-byte loads
#pragma unroll
      for (int v = 0; v < 6; ++v) {
        const float4 q = __ldg((const float4 *)rp + v);
        r[4 * v] = q.x;
        r[4 * v + 1] = q.y;
        r[4 * v + 2] = q.z;
        r[4 * v + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int a = 0; a < 24; a += 2) {
        const double2 q = __ldg((const double2 *)(rp + a));
        r[a] = q.x;
        r[a + 1] = q.y;
      }
    }
    T s0 = 0., s1 = 0.;
#pragma unroll
    for (int a = 0; a < 9; ++a) {
      s0 += r[2 * a] * (T)dc[a];
      s1 += r[2 * a + 1] * (T)dc[a];
    }
    a0 += r[18] * s0 + r[21] * s1;
    a1 += r[19] * s0 + r[22] * s1;
    a2 += r[20] * s0 + r[23] * s1;
  }
  a0 = grp_sum(a0);
  a1 = grp_sum(a1);
  a2 = grp_sum(a2);
  if (ln == 0 && valid) {
    const T *pv = Store<T>::ptV(L) + (size_t)p * PREC;
    double *xo = L.x + L.nrioff + 3 * p;
    if constexpr (sizeof(T) == 8) {
      const T r0 = pv[9] - a0, r1 = pv[10] - a1, r2 = pv[11] - a2;
      xo[0] = pv[0] * r0 + pv[1] * r1 + pv[2] * r2;
      xo[1] = pv[3] * r0 + pv[4] * r1 + pv[5] * r2;
      xo[2] = pv[6] * r0 + pv[7] * r1 + pv[8] * r2;
    } else {
      // whitened: a = L^-1 sum G^T Bc dc, dX = L^-T (q - a)
      const double y0 = (double)pv[9] - a0, y1 = (double)pv[10] - a1, y2 = (double)pv[11] - a2;
      xo[0] = (double)pv[0] * y0 + (double)pv[3] * y1 + (double)pv[6] * y2;
      xo[1] = (double)pv[4] * y1 + (double)pv[7] * y2;
      xo[2] = (double)pv[8] * y2;
    }
  }
}

// Camera entries of the step: x[k] = (float) exiv (rbacore.cpp:1181-1186).
__global__ void k_xcam(DevLSA L, const double *__restrict__ xsol) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = i / 9 + L.begini, a = i % 9;
  if (k >= L.nimg) return;
  const int cp = L.camparv[k], np = L.camparv[k + 1] - cp;
  if (a < np) L.x[cp + a] = (double)(float)xsol[(size_t)k * 9 + a];
}

// XPMatricesnew = XPMatrices - x with the NaN/Inf check (rbacore.cpp:541-548).
__global__ void k_update(DevLSA L, int nunk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nunk) return;
  const double v = L.x[i];
  if (!isfinite(v)) atomicOr(L.err, 1);
  L.XPMn[i] = L.XPM[i] - v;
}

// ------------------------------------------------- camera (de)coding
// DecodeCameras, rbacore.cpp:1733-1800.
__global__ void k_decode(DevLSA L, const double *__restrict__ XM) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L.nimg) return;
  // a NaN step returns before DecodeCameras (rbacore.cpp:541-550): keep the
  // previous trial cameras, which OutputLSAc reports
  if (*(volatile int *)L.err & 1) return;
  CamState &c = L.camn[k];
  if (k == 0 && !L.ao) {
    int a = -1;
    if (L.addmask & 1) c.d0 = XM[++a];
    if (L.addmask & 2) c.d1 = XM[++a];
    if (L.addmask & 4) c.K00 = c.K11 = XM[++a];
    return;
  }
  const int cp = L.camparv[k];
  double Ra[9];
  cayley(XM[cp], XM[cp + 1], XM[cp + 2], Ra);
  const double *B = L.Rb + (size_t)k * 9;
  double R[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) R[i * 3 + j] = Ra[i * 3] * B[j] + Ra[i * 3 + 1] * B[3 + j] + Ra[i * 3 + 2] * B[6 + j];
  rectify(R, 3);
#pragma unroll
  for (int i = 0; i < 9; ++i) c.R[i] = R[i];
  double e[3];
  if (k == L.normcamera) {
    e[L.gauge[0]] = XM[cp + 3];
    e[L.gauge[1]] = XM[cp + 4];
    e[L.gauge[2]] = 0.;
  } else {
    e[0] = XM[cp + 3];
    e[1] = XM[cp + 4];
    e[2] = XM[cp + 5];
  }
  const double *pb = L.PCb + (size_t)k * 3;
  c.PC[0] = e[0] + pb[0];
  c.PC[1] = e[1] + pb[1];
  c.PC[2] = e[2] + pb[2];
  int a = k == L.normcamera ? 4 : 5;
  if (L.addmask & 1) c.d0 = XM[++a + cp];
  if (L.addmask & 2) c.d1 = XM[++a + cp];
  if (L.addmask & 4) c.K00 = c.K11 = XM[++a + cp];
}

// EncodeCameras, rbacore.cpp:999-1087.
__global__ void k_encode(DevLSA L) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= L.nimg) return;
  if (k == 0 && !L.ao) {
    int a = -1;
    if (L.addmask & 1) L.XPM[++a] = L.dc[0];
    if (L.addmask & 2) L.XPM[++a] = L.dc[1];
    if (L.addmask & 4) L.XPM[++a] = L.Kc[0];
    return;
  }
  double *P = L.Pacc + (size_t)k * 12;
  rectify(P, 4);
  double *R = L.Rb + (size_t)k * 9;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) R[r * 3 + c] = P[r * 4 + c];
  double *pc = L.PCb + (size_t)k * 3;
  for (int i = 0; i < 3; ++i) pc[i] = R[i] * P[3] + R[3 + i] * P[7] + R[6 + i] * P[11];
  const int cp = L.camparv[k];
  L.XPM[cp] = L.XPM[cp + 1] = L.XPM[cp + 2] = 0.;
  int a;
  if (k == L.normcamera) {
    float maxv = 0.f;
    int maxi = 0;
    for (int i = 0; i < 3; ++i)
      if (fabs(pc[i]) > (double)maxv) {
        maxv = (float)fabs(pc[i]);
        maxi = i;
      }
    int ii = 0;
    for (int i = 0; i < 3; ++i)
      if (i != maxi) L.gauge[ii++] = i;
    L.gauge[2] = maxi;
    L.XPM[cp + 3] = L.XPM[cp + 4] = 0.;
    a = 4 + cp;
  } else {
    L.XPM[cp + 3] = L.XPM[cp + 4] = L.XPM[cp + 5] = 0.;
    a = 5 + cp;
  }
  if (L.addmask & 1) L.XPM[++a] = L.dc[2 * k];
  if (L.addmask & 2) L.XPM[++a] = L.dc[2 * k + 1];
  if (L.addmask & 4) L.XPM[++a] = L.Kc[9 * k];
}

// StoreResultsIteration, rbacore.cpp:891-918.
__global__ void k_store(DevLSA L, int xpmsize) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < xpmsize) L.XPM[i] = L.XPMn[i];
  if (i < L.nobs) L.o_flagnew[i] = L.o_flag[i];
  if (i < L.nimg) {
    const CamState &c = L.camn[i];
    double *P = L.Pacc + (size_t)i * 12;
    for (int r = 0; r < 3; ++r) {
      for (int cc = 0; cc < 3; ++cc) P[r * 4 + cc] = c.R[r * 3 + cc];
      P[r * 4 + 3] = c.R[r * 3] * c.PC[0] + c.R[r * 3 + 1] * c.PC[1] + c.R[r * 3 + 2] * c.PC[2];
    }
    double *K = L.Kc + (size_t)i * 9;
    K[0] = c.K00;
    K[1] = c.K01;
    K[2] = c.K02;
    K[4] = c.K11;
    K[5] = c.K12;
    K[8] = 1.;
    L.dc[2 * i] = c.d0;
    L.dc[2 * i + 1] = c.d1;
  }
}

// PrepareWeights2D (rbacore.cpp:704-783): Wij = Wijold and the terms of
// the float weight sum.
__global__ void k_prepare_weights(DevLSA L) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.nobs) return;
  const float4 w = L.o_wold[i];
  L.o_w[i] = w;
  L.o_wterm[i] = __fadd_rn(w.x, w.y);
  L.o_flag[i] = 0;
  L.o_flagnew[i] = 0;
}

// ----------------------------------------------------------- reweight
// Reweight2D, rbacore.cpp:823-887.
__global__ void k_rw_vals(DevLSA L, float *vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.nobs) return;
  const int o = L.camlist[i];
  const int p = L.o_pt[o];
  int pxs = (L.pt_off[p + 1] - L.pt_off[p]) * 2;
  if (pxs < 4) pxs = 4;
  const float rf = __fdiv_rn((float)pxs, (float)(pxs - 3));
  const float redfac = __fmul_rn(rf, rf);
  vals[i] = __fmul_rn(L.o_s0rmv[o], redfac);
}

// Per-image median by an exact radix select on the float bit patterns
// (values are >= 0, so the unsigned order is the numeric order).
__global__ void __launch_bounds__(256) k_median(DevLSA L, const float *vals, float *sig00v, int iflag) {
  const int k = blockIdx.x;
  if (k >= L.nimg) return;
  const int beg = L.coff[k], end = L.coff[k + 1], n = end - beg;
  __shared__ unsigned hist[256];
  __shared__ unsigned s_prefix, s_mask;
  __shared__ int s_rank;
  if (threadIdx.x == 0) {
    s_prefix = 0u;
    s_mask = 0u;
    s_rank = n / 2;
  }
  __syncthreads();
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    hist[threadIdx.x] = 0u;
    __syncthreads();
    const unsigned prefix = s_prefix, mask = s_mask;
    for (int i = beg + threadIdx.x; i < end; i += blockDim.x) {
      unsigned key = __float_as_uint(vals[i]);
      if (key == 0x80000000u) key = 0u;
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int r = s_rank;
      unsigned b = 0;
      for (; b < 256; ++b) {
        if ((int)hist[b] > r) break;
        r -= (int)hist[b];
      }
      if (b > 255) b = 255;
      s_rank = r;
      s_prefix = prefix | (b << shift);
      s_mask = mask | (255u << shift);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float med = n > 0 ? __uint_as_float(s_prefix) : 0.f;
    float s = __fdiv_rn(1.f, __fmul_rn(med, 2.1981f));
    if (iflag > 1) s = __fmul_rn(s, 0.001f);
    sig00v[k] = s;
  }
}

__global__ void k_rw_apply(DevLSA L, const float *sig00v, int *nflag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int f = 0;
  if (i < L.nobs) {
    float ww = __fmul_rn(L.o_s0rmv[i], sig00v[L.o_cam[i]]);
    const bool fl = ww > 9.f;
    L.o_flag[i] = fl ? 1 : 0;
    if (fl) {
      ww = 1.e-4f;
      f = 1;
    } else {
      ww = 1.f;
    }
    const float4 wo = L.o_wold[i];
    float4 w;
    w.x = __fmul_rn(ww, wo.x);
    w.y = __fmul_rn(ww, wo.y);
    w.z = __fmul_rn(ww, wo.z);
    w.w = 0.f;
    if (__fadd_rn(w.x, w.y) < 2.e-8f) {
      w.x = w.y = 1.e-8f;
      w.z = 0.f;
    }
    L.o_w[i] = w;
    L.o_wterm[i] = __fadd_rn(w.x, w.y);
  }
  f = __syncthreads_count(f);
  if (threadIdx.x == 0 && f) atomicAdd(nflag, f);
}

// ------------------------------------------------------ final cost
// FP64 cost and squared residual sum of the accepted state with the
// Exteval projection (P X, distortion, f): the shared evaluator the oracle
// uses too.
__global__ void k_final_cost(DevLSA L, double *partials) {
  __shared__ double sc[256], sq[256];
  double c = 0., q = 0.;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L.nobs; i += gridDim.x * blockDim.x) {
    const int k = L.o_cam[i], p = L.o_pt[i];
    const double *M = L.Pacc + (size_t)k * 12;
    const double *X = L.XPM + L.nrioff + 3 * p;
    double p1 = M[0] * X[0] + M[1] * X[1] + M[2] * X[2] + M[3];
    double p2 = M[4] * X[0] + M[5] * X[1] + M[6] * X[2] + M[7];
    double p3 = M[8] * X[0] + M[9] * X[1] + M[10] * X[2] + M[11];
    if (fabs(p3) < 1.e-3)
      p3 = p3 > 0. ? 1.e3 : -1.e3;
    else
      p3 = 1. / p3;
    p1 *= p3;
    p2 *= p3;
    const double dist = p1 * p1 + p2 * p2;
    const double z = 1. + (L.dc[2 * k] * dist + L.dc[2 * k + 1] * dist * dist);
    p1 *= z * L.Kc[9 * k];
    p2 *= z * L.Kc[9 * k];
    const float2 xg = L.o_xg[i];
    const double dx = (double)xg.x - p1, dy = (double)xg.y - p2;
    const float4 w = L.o_wold[i];
    c += dx * dx * w.x + dy * dy * w.y + 2. * dx * dy * w.z;
    q += dx * dx + dy * dy;
  }
  sc[threadIdx.x] = c;
  sq[threadIdx.x] = q;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sc[threadIdx.x] += sc[threadIdx.x + s];
      sq[threadIdx.x] += sq[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = sc[0];
    partials[2 * blockIdx.x + 1] = sq[0];
  }
}

// A track entry that names no observation sets *bad (Exteval, refinement).
__global__ void k_check_tracks(int nt, int n, const int *__restrict__ pt_img, const int *__restrict__ pt_slot,
                               const int *__restrict__ img_off, int *bad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int im = pt_img[t], sl = pt_slot[t];
  if (im < 0 || im >= n || sl < 0 || sl >= img_off[im + 1] - img_off[im]) *bad = 1;
}

// ------------------------------------------------------------ Exteval
// EvalLSA + CalcCorrPointMulti (rpbacore.cpp:778-837, 882-941): one thread
// per point, float sums in the reference's order within the point.
__global__ void k_exteval(int n_points, const int *__restrict__ pt_off, const int *__restrict__ pt_img,
                          const int *__restrict__ pt_slot, const int *__restrict__ img_off,
                          const float *__restrict__ pmat, const float *__restrict__ Kf,
                          const float *__restrict__ dist, const float *__restrict__ XX,
                          const float *__restrict__ xg, const float *__restrict__ wx,
                          const float *__restrict__ wy, const float *__restrict__ wxy, double *resid,
                          float *ptterm, int *ptred) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_points) return;
  const int s = pt_off[p], e = pt_off[p + 1];
  const int n = e - s;
  for (int j = s; j < e; ++j) resid[2 * j] = resid[2 * j + 1] = 0.;
  if (n <= 1) {
    ptterm[p] = 0.f;
    ptred[p] = 0;
    return;
  }
  float wsum = 0.f;
  for (int j = s; j < e; ++j) {
    const int sl = img_off[pt_img[j]] + pt_slot[j];
    wsum = __fadd_rn(wsum, __fadd_rn(wx[sl], wy[sl]));
  }
  wsum = __fdiv_rn(wsum, (float)(2 * n));
  const double X0 = XX[3 * p], X1 = XX[3 * p + 1], X2 = XX[3 * p + 2];
  float sig0 = 0.f;
  for (int j = s; j < e; ++j) {
    const int im = pt_img[j];
    const int sl = img_off[im] + pt_slot[j];
    const float *P = pmat + 12 * im;
    double p1 = add(add(add(mul((double)P[0], X0), mul((double)P[1], X1)), mul((double)P[2], X2)), (double)P[3]);
    double p2 = add(add(add(mul((double)P[4], X0), mul((double)P[5], X1)), mul((double)P[6], X2)), (double)P[7]);
    double p3 = add(add(add(mul((double)P[8], X0), mul((double)P[9], X1)), mul((double)P[10], X2)), (double)P[11]);
    if (fabs(p3) < 1.e-3)
      p3 = p3 > 0. ? 1.e3 : -1.e3;
    else
      p3 = __ddiv_rn(1., p3);
    p1 = mul(p1, p3);
    p2 = mul(p2, p3);
    const double dd = add(mul(p1, p1), mul(p2, p2));
    const double z = add(1., add(mul((double)dist[2 * im], dd), mul(mul((double)dist[2 * im + 1], dd), dd)));
    p1 = mul(p1, z);
    p2 = mul(p2, z);
    p1 = mul(p1, (double)Kf[9 * im]);
    p2 = mul(p2, (double)Kf[9 * im]);
    const double dx = sub((double)xg[2 * sl], p1), dy = sub((double)xg[2 * sl + 1], p2);
    resid[2 * j] = dx;
    resid[2 * j + 1] = dy;
    const double t = add(add(mul(mul(dx, dx), (double)wx[sl]), mul(mul(dy, dy), (double)wy[sl])),
                         mul(mul(mul(2., dx), dy), (double)wxy[sl]));
    sig0 = __fadd_rn(sig0, (float)t);
  }
  ptterm[p] = __fdiv_rn(sig0, wsum);
  ptred[p] = 2 * n - 3;
}

// ------------------------------------------------------ RobustDelete
// rbacore.cpp:922-995: observations flagged at the last accepted step are
// erased; a point left with fewer than minimagenrdel observations goes.
__global__ void k_delete_mark(DevLSA L, int *okeep, int *pkeep) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= L.npts) return;
  const int t0 = L.pt_off[p], t1 = L.pt_off[p + 1];
  int nf = 0;
  for (int o = t0; o < t1; ++o) nf += L.o_flagnew[o] ? 1 : 0;
  const bool erase = nf > 0 && (t1 - t0 - nf) < L.minimagenrdel;
  pkeep[p] = erase ? 0 : 1;
  for (int o = t0; o < t1; ++o) okeep[o] = (!erase && !L.o_flagnew[o]) ? 1 : 0;
}

__global__ void k_delete_obs(DevLSA L, const int *oidx, const int *pidx, const int *okeep, int *o_cam_n,
                             int *o_slot_n, int *o_pt_n, float2 *o_xg_n, float4 *o_wold_n) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= L.nobs || !okeep[o]) return;
  const int q = oidx[o];
  o_cam_n[q] = L.o_cam[o];
  o_slot_n[q] = L.o_slot[o];
  o_pt_n[q] = pidx[L.o_pt[o]];
  o_xg_n[q] = L.o_xg[o];
  o_wold_n[q] = L.o_wold[o];
}

__global__ void k_delete_pts(DevLSA L, const int *oidx, const int *pidx, const int *pkeep, int nobs_new,
                             int npts_new, int *pt_off_n, int *pt_id_n, double *X_n) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p == 0) pt_off_n[npts_new] = nobs_new;
  if (p >= L.npts || !pkeep[p]) return;
  const int q = pidx[p];
  pt_id_n[q] = L.pt_id[p];
  pt_off_n[q] = oidx[L.pt_off[p]];
  const double *X = L.XPM + L.nrioff + 3 * p;
  X_n[3 * q] = X[0];
  X_n[3 * q + 1] = X[1];
  X_n[3 * q + 2] = X[2];
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_cost(const DevLSA &L, const double *XM, bool srmv, cudaStream_t s) {
  if (L.nobs > 0) k_cost<<<nblk(L.nobs, 256), 256, 0, s>>>(L, XM, srmv ? 1 : 0);
}

void launch_seq_sum(const float *v, int n, float *out, cudaStream_t s) {
  k_seq_sum<<<1, SS_T, 0, s>>>(v, n, out);
}

template <class T>
static void point_pass(const DevLSA &L, double multfact1, cudaStream_t s) {
  constexpr int W = PointGeom<T>::W;
  static_assert(W * sizeof(PointShared<T>) <= 48 * 1024, "shared memory without an attribute");
  k_point<T><<<nblk(L.npts, PT_N * W), 32 * W, W * sizeof(PointShared<T>), s>>>(L, multfact1);
}

void launch_point_pass(const DevLSA &L, double multfact1, cudaStream_t s) {
  if (L.npts <= 0) return;
  if (L.rec32)
    point_pass<float>(L, multfact1, s);
  else
    point_pass<double>(L, multfact1, s);
}

void launch_camera_pass(const DevLSA &L, double multfact1, cudaStream_t s) {
  const int nc = L.nimg - L.begini;
  if (nc <= 0) return;
  if (L.rec32)
    k_camera<float><<<nc, 32 * CAM_W, 0, s>>>(L, multfact1);
  else
    k_camera<double><<<nc, 32 * CAM_W, 0, s>>>(L, multfact1);
}

void launch_pair_pass(const DevLSA &L, cudaStream_t s) {
  if (L.nboff <= 0) return;
  if (L.rec32)
    k_pair<float><<<nblk(L.nboff, PAIR_W), 32 * PAIR_W, 0, s>>>(L);
  else
    k_pair<double><<<nblk(L.nboff, PAIR_W), 32 * PAIR_W, 0, s>>>(L);
}

void launch_backsub(const DevLSA &L, const double *xsol, cudaStream_t s) {
  if (L.npts <= 0) return;
  if (L.rec32)
    k_backsub<float><<<nblk((long long)L.npts * GRP, 128), 128, 0, s>>>(L, xsol);
  else
    k_backsub<double><<<nblk((long long)L.npts * GRP, 128), 128, 0, s>>>(L, xsol);
}

void launch_xcam(const DevLSA &L, const double *xsol, cudaStream_t s) {
  const int n = (L.nimg - L.begini) * 9;
  if (n > 0) k_xcam<<<nblk(n, 256), 256, 0, s>>>(L, xsol);
}

void launch_update(const DevLSA &L, int nunk, cudaStream_t s) {
  if (nunk > 0) k_update<<<nblk(nunk, 256), 256, 0, s>>>(L, nunk);
}

void launch_decode(const DevLSA &L, const double *XM, cudaStream_t s) {
  k_decode<<<nblk(L.nimg, 128), 128, 0, s>>>(L, XM);
}

void launch_encode(const DevLSA &L, cudaStream_t s) { k_encode<<<nblk(L.nimg, 128), 128, 0, s>>>(L); }

void launch_store(const DevLSA &L, int xpmsize, cudaStream_t s) {
  long long n = xpmsize;
  if (L.nobs > n) n = L.nobs;
  if (L.nimg > n) n = L.nimg;
  k_store<<<nblk(n, 256), 256, 0, s>>>(L, xpmsize);
}

void launch_prepare_weights(const DevLSA &L, cudaStream_t s) {
  if (L.nobs > 0) k_prepare_weights<<<nblk(L.nobs, 256), 256, 0, s>>>(L);
}

void launch_reweight(const DevLSA &L, int iflag, float *vals, float *sig00v, int *nflag, cudaStream_t s) {
  cudaMemsetAsync(nflag, 0, sizeof(int), s);
  if (L.nobs > 0) k_rw_vals<<<nblk(L.nobs, 256), 256, 0, s>>>(L, vals);
  k_median<<<L.nimg, 256, 0, s>>>(L, vals, sig00v, iflag);
  if (L.nobs > 0) k_rw_apply<<<nblk(L.nobs, 256), 256, 0, s>>>(L, sig00v, nflag);
}

void launch_final_cost(const DevLSA &L, double *partials, int nparts, cudaStream_t s) {
  k_final_cost<<<nparts, 256, 0, s>>>(L, partials);
}

void launch_gcp_cost(const DevLSA &L, const double *XM, float *out, cudaStream_t s) {
  if (L.npts > 0) k_gcp_cost<<<nblk(L.npts, 256), 256, 0, s>>>(L, XM, out);
}

void launch_check_tracks(int nt, int n, const int *pt_img, const int *pt_slot, const int *img_off, int *bad,
                         cudaStream_t s) {
  if (nt > 0) k_check_tracks<<<nblk(nt, 256), 256, 0, s>>>(nt, n, pt_img, pt_slot, img_off, bad);
}

void launch_exteval(int n_points, const int *pt_off, const int *pt_img, const int *pt_slot, const int *img_off,
                    const float *pmat, const float *K, const float *dist, const float *XX, const float *xg,
                    const float *wx, const float *wy, const float *wxy, double *resid, float *ptterm,
                    int *ptred, cudaStream_t s) {
  if (n_points > 0)
    k_exteval<<<nblk(n_points, 128), 128, 0, s>>>(n_points, pt_off, pt_img, pt_slot, img_off, pmat, K, dist, XX,
                                                  xg, wx, wy, wxy, resid, ptterm, ptred);
}

void launch_delete_mark(const DevLSA &L, int *okeep, int *pkeep, cudaStream_t s) {
  if (L.npts > 0) k_delete_mark<<<nblk(L.npts, 256), 256, 0, s>>>(L, okeep, pkeep);
}

void launch_delete_compact(const DevLSA &L, const int *oidx, const int *pidx, const int *okeep, const int *pkeep,
                           int nobs_new, int npts_new, int *o_cam_n, int *o_slot_n, int *o_pt_n, float2 *o_xg_n,
                           float4 *o_wold_n, int *pt_off_n, int *pt_id_n, double *X_n, cudaStream_t s) {
  if (L.nobs > 0)
    k_delete_obs<<<nblk(L.nobs, 256), 256, 0, s>>>(L, oidx, pidx, okeep, o_cam_n, o_slot_n, o_pt_n, o_xg_n,
                                                   o_wold_n);
  k_delete_pts<<<nblk(L.npts > 0 ? L.npts : 1, 256), 256, 0, s>>>(L, oidx, pidx, pkeep, nobs_new, npts_new,
                                                                  pt_off_n, pt_id_n, X_n);
}

}  // namespace rpba
