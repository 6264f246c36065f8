// exactsum.cu -- the reference's float accumulations (sig0 += term in
// rbacore.cpp:1327, wsum += w in :727 and :881), computed in parallel with a
// result bitwise equal to the sequential float loop.
//
// Method.  Let s be the running float sum, s in [2^E, 2^(E+1)), u = ulp(s) =
// 2^(E-23), S = s/u (an integer in [2^23, 2^24)).  For v >= 0 with
// S + floor(v/u) < 2^24 the float addition is fl(s + v) = s + u*rne(v/u)
// with rne(v/u) = floor(v/u) + [frac > 1/2], except when v/u is exactly
// halfway between integers (a tie): then round-half-even gives
// floor(v/u) + [S + floor(v/u) odd], and the new S is even.  So inside one
// binade each element acts on the parity p of the running integer sum as a
// two-state transform  p -> (increment r(p), new parity q(p)), and a run of
// elements is the composition of their transforms, an associative operation:
// scans of per-thread, per-warp and per-CTA composites give every prefix
// without a sequential pass, ties included.  A run ends only at the first
// element k with S + R_(k-1) + floor(v_k/u) >= 2^24 (the sum leaves the
// binade); that element is added with a real float addition and a new run
// starts in the new binade.  Runs are few: the sum leaves a binade only when
// it doubles.  Each step of the scan covers a window, the elements from the
// run's start on, as many again as the sum has taken so far: the sum doubles
// inside it unless the terms shrink (then the next step takes the next
// window in the same binade), so the steps together read the input about
// twice instead of once per binade.
//
// A step is latency: a scan over the window's composites, the search for the
// crossing element, and in the grid form one barrier and one published word.
// So the first ES_SOLO elements are summed by one CTA (its steps are two
// block barriers each), inputs up to that length by a kernel of one CTA, not
// cooperative; longer ones go on with one CTA per SM.  Measured (18 to 20
// sums a solve): 5.4k terms 82 -> 22 us, 30k 115 -> 37 us, 0.87M 277 ->
// 102 us, 28M 704 -> 216 us; before, the first 2,048 elements were added
// at 25 cycles each, a step took four grid barriers, and one thread walked
// the chunks' composites.
//
// The first HEAD elements and any stretch where s is zero or subnormal are
// added by one warp in plain sequence.  Inputs must be finite and >= 0.
#include <cuda.h>

#include <climits>
#include <mutex>

#include "../../include/rpba_b200.h"
#include "gridsync.cuh"
#include "internal.h"

namespace rpba {

namespace {

constexpr int ES_T = 1024;
constexpr int ES_W = ES_T / 32;
constexpr int HEAD = 512;        // elements added in plain sequence
constexpr int ES_SEQ = 1024;     // elements per sequential block at most
constexpr int ES_WMIN = 2048;    // smallest window of a run step
constexpr int ES_SOLO = 65536;   // elements one CTA sums (a solo step past it costs more than a grid step)
constexpr int ES_MAXG = 256;     // CTAs at most (eight composites a lane)
constexpr int MAX_SEGMENTS = 512;
// Increments saturate here: a run crosses its binade long before (at 2^24),
// and nothing past the first crossing is used.
constexpr int SAT = 1 << 26;
constexpr int TOP = 1 << 24;

// Composite transform of a run of elements for incoming parity 0 and 1:
// total increment R, M = max over the run of (increment before the element +
// floor(v/u)), the crossing test (-1: no element), and the outgoing parities
// (bit p of q).
struct Xf {
  int R0, R1, M0, M1;
  unsigned q;
};
__device__ __forceinline__ Xf xf_identity() { return Xf{0, 0, -1, -1, 2u}; }
// a then b
__device__ __forceinline__ Xf xf_then(const Xf &a, const Xf &b) {
  const bool m0 = a.q & 1u, m1 = a.q & 2u;
  const int bM0 = m0 ? b.M1 : b.M0, bM1 = m1 ? b.M1 : b.M0;
  Xf x;
  x.R0 = min(a.R0 + (m0 ? b.R1 : b.R0), SAT);
  x.R1 = min(a.R1 + (m1 ? b.R1 : b.R0), SAT);
  x.M0 = max(a.M0, bM0 < 0 ? -1 : min(a.R0 + bM0, SAT));
  x.M1 = max(a.M1, bM1 < 0 ? -1 : min(a.R1 + bM1, SAT));
  x.q = ((b.q >> (m0 ? 1 : 0)) & 1u) | (((b.q >> (m1 ? 1 : 0)) & 1u) << 1);
  return x;
}
__device__ __forceinline__ Xf xf_up(const Xf &a, int o) {
  Xf x;
  x.R0 = __shfl_up_sync(0xffffffffu, a.R0, o);
  x.R1 = __shfl_up_sync(0xffffffffu, a.R1, o);
  x.M0 = __shfl_up_sync(0xffffffffu, a.M0, o);
  x.M1 = __shfl_up_sync(0xffffffffu, a.M1, o);
  x.q = __shfl_up_sync(0xffffffffu, a.q, o);
  return x;
}
// Inclusive scan over the warp's lanes, in lane order.
__device__ __forceinline__ Xf xf_scan(Xf x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Xf u = xf_up(x, o);
    if (lane >= o) x = xf_then(u, x);
  }
  return x;
}
__device__ __forceinline__ Xf xf_exclusive(const Xf &incl, int lane) {
  const Xf u = xf_up(incl, 1);
  return lane == 0 ? xf_identity() : u;
}

// The binade of a normal s: unit u, v -> v / u as two exact float factors
// (powers of two whose product can be outside the float range), S = s / u.
struct Binade {
  float s1, s2;
  int S;
  double u;
};
__device__ __forceinline__ Binade binade_of(float s) {
  Binade b;
  int E;
  frexpf(s, &E);
  E -= 1;  // s in [2^E, 2^(E+1))
  const int k = 23 - E, k1 = k / 2;
  b.s1 = ldexpf(1.f, k1);
  b.s2 = ldexpf(1.f, k - k1);
  b.S = (int)((s * b.s1) * b.s2);
  b.u = ldexp(1.0, E - 23);
  return b;
}
__device__ __forceinline__ float binade_value(const Binade &b, int S) { return (float)((double)S * b.u); }

// floor(v/u), rne(v/u) away from ties, and whether v/u is a tie; past the
// saturation (or not a number) the element crosses in any case.
__device__ __forceinline__ void classify(float v, const Binade &b, int &fl, int &r, bool &tie) {
  const float f = (v * b.s1) * b.s2;
  if (!(f < (float)SAT)) {
    fl = r = SAT;
    tie = false;
    return;
  }
  const float ff = floorf(f), fr = f - ff;
  fl = (int)ff;
  tie = fr == 0.5f;
  r = fl + (fr > 0.5f ? 1 : 0);
}

// Apply one element to a composite (both incoming parities).
__device__ __forceinline__ void xf_push(Xf &x, int fl, int r, bool tie) {
  const int r0 = tie ? fl + (((int)(x.q & 1u) + fl) & 1) : r;
  const int r1 = tie ? fl + (((int)(x.q >> 1) + fl) & 1) : r;
  x.M0 = max(x.M0, min(x.R0 + fl, SAT));
  x.M1 = max(x.M1, min(x.R1 + fl, SAT));
  x.R0 = min(x.R0 + r0, SAT);
  x.R1 = min(x.R1 + r1, SAT);
  x.q ^= (unsigned)(r0 & 1) | ((unsigned)(r1 & 1) << 1);
}

// Four elements onto a composite whose two parities have not parted (R0, M0
// stand for both), unless one of them is a tie or saturates: 10 instead of 25
// instructions an element.  Increments are not negative, so the saturation of
// R and M can wait for the end of the group.
__device__ __forceinline__ bool xf_push4(Xf &x, const float4 &a, const Binade &b) {
  const float f0 = (a.x * b.s1) * b.s2, f1 = (a.y * b.s1) * b.s2, f2 = (a.z * b.s1) * b.s2, f3 = (a.w * b.s1) * b.s2;
  const float g0 = floorf(f0), g1 = floorf(f1), g2 = floorf(f2), g3 = floorf(f3);
  const float h0 = f0 - g0, h1 = f1 - g1, h2 = f2 - g2, h3 = f3 - g3;
  const bool in = f0 < (float)SAT && f1 < (float)SAT && f2 < (float)SAT && f3 < (float)SAT;
  if (!in || h0 == 0.5f || h1 == 0.5f || h2 == 0.5f || h3 == 0.5f) return false;
  const int R0 = x.R0, R1 = R0 + (int)g0 + (h0 > 0.5f), R2 = R1 + (int)g1 + (h1 > 0.5f), R3 = R2 + (int)g2 + (h2 > 0.5f),
            R4 = R3 + (int)g3 + (h3 > 0.5f);
  const int M = max(max(R0 + (int)g0, R1 + (int)g1), max(R2 + (int)g2, R3 + (int)g3));
  x.M0 = max(x.M0, min(M, SAT));
  x.R0 = min(R4, SAT);
  if ((R4 - R0) & 1) x.q ^= 3u;
  return true;
}

// Composite of v[lo, hi): 16-byte loads of whole aligned groups.
__device__ __forceinline__ Xf xf_range(const float *__restrict__ v, int lo, int hi, bool aligned, const Binade &b) {
  Xf x = xf_identity();
  bool parted = false;
  auto push = [&](float a) {
    int fl, r;
    bool tie;
    classify(a, b, fl, r, tie);
    if (!parted) {
      x.R1 = x.R0;
      x.M1 = x.M0;
      parted = true;
    }
    xf_push(x, fl, r, tie);
  };
  auto push4 = [&](const float4 &a) {
    if (!parted && xf_push4(x, a, b)) return;
    push(a.x);
    push(a.y);
    push(a.z);
    push(a.w);
  };
  int k = lo;
  if (aligned) {
    for (; k < hi && (k & 3); ++k) push(__ldg(v + k));
    for (; k + 16 <= hi; k += 16) {
      float4 a[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) a[m] = __ldg((const float4 *)(v + k) + m);
#pragma unroll
      for (int m = 0; m < 4; ++m) push4(a[m]);
    }
    for (; k + 4 <= hi; k += 4) push4(__ldg((const float4 *)(v + k)));
  }
  for (; k < hi; ++k) push(__ldg(v + k));
  if (!parted) {
    x.R1 = x.R0;
    x.M1 = x.M0;
  }
  return x;
}

// Adds v[k..) onto the state (R, q) up to the element that crosses, then that
// element with a float addition.
__device__ __forceinline__ void cross_element(const float *__restrict__ v, int lo, int hi, int n, const Binade &b,
                                              int R, int q, float &s, int &i) {
  for (int k = lo; k < hi; ++k) {
    int fl, r;
    bool tie;
    classify(__ldg(v + k), b, fl, r, tie);
    if (b.S + R + fl >= TOP) {
      s = __fadd_rn(binade_value(b, b.S + R), __ldg(v + k));
      i = isfinite(s) ? k + 1 : n;
      return;
    }
    const int rr = tie ? fl + ((q + fl) & 1) : r;
    R += rr;
    q = (q + rr) & 1;
  }
}

struct __align__(16) EsShared {
  float buf[ES_SEQ];  // first: read 16 bytes at a time
  Xf w[ES_W];         // the warps' composites
  float s;
  int i;
  int R, q;           // grid step: the state before the chunk that crosses
  int cx;             // grid step: the chunk that crosses, or -1
};

// v[i, i + cnt) added in plain sequence onto s by warp 0 (cnt <= ES_SEQ); the
// values are staged in shared memory, so the chain is the additions alone.
// Valid in warp 0.
__device__ __forceinline__ float seq_block(const float *__restrict__ v, int i, int cnt, float s, float *buf) {
  __syncthreads();
  for (int j = threadIdx.x; j < cnt; j += blockDim.x) buf[j] = __ldg(v + i + j);
  __syncthreads();
  if (threadIdx.x < 32) {
    int j = 0;
#pragma unroll 4
    for (; j + 4 <= cnt; j += 4) {
      const float4 a = *(const float4 *)(buf + j);
      s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
    }
    for (; j < cnt; ++j) s = __fadd_rn(s, buf[j]);
  }
  return s;
}

// The window [i0, wend) cut into `parts` pieces at multiples of four, and
// thread tid's range of piece `part`.
__device__ __forceinline__ void thread_range(int i0, int wend, int part, int parts, int &lo, int &hi, int least = 4) {
  const int base = i0 & ~3;
  const int per = max(least, (((wend - base + parts - 1) / parts + ES_T - 1) / ES_T + 3) & ~3);
  const long long a = (long long)base + ((long long)part * ES_T + threadIdx.x) * per;
  lo = (int)max((long long)i0, min(a, (long long)wend));
  hi = (int)min(a + per, (long long)wend);
}

// Sums from the front until at least `stop` elements are taken (or n) and s
// is normal; the state is left in sh.s, sh.i.
__device__ void es_solo(const float *__restrict__ v, int n, int stop, bool aligned, EsShared &sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float s = 0.f;
  int i = 0;
  for (int seg = 0;; ++seg) {
    // plain sequence: the head, the zero and subnormal range, and past
    // MAX_SEGMENTS steps (far more than sums of real data take) the rest
    while (i < n && (i < HEAD || !(s >= 1.17549435e-38f) || seg >= MAX_SEGMENTS)) {
      const int cnt = min(n - i, i < HEAD ? HEAD - i : ES_SEQ);
      const float t = seq_block(v, i, cnt, s, sh.buf);
      if (tid == 0) sh.s = t;
      __syncthreads();
      s = sh.s;
      i = isfinite(s) ? i + cnt : n;
    }
    if (i >= n || i >= stop) break;
    const Binade b = binade_of(s);
    const int p0 = b.S & 1;
    const int wend = (int)min((long long)n, (long long)i + max(i, ES_WMIN));
    // (a short window goes to the first warps alone, eight elements a thread
    // at least, and one warp looks for the crossing: 32 warps that all scan
    // spent most of a step's 4,400 cycles on issuing the scans)
    int lo, hi;
    thread_range(i, wend, 0, 1, lo, hi, 8);
    Xf tx = xf_identity(), incl = tx;
    if (__any_sync(0xffffffffu, lo < hi)) {
      tx = xf_range(v, lo, hi, aligned, b);
      incl = xf_scan(tx, lane);
    }
    if (lane == 31) sh.w[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      // the state before each warp, and the first that crosses
      const Xf wx = sh.w[lane];
      const Xf wi = xf_scan(wx, lane), we = xf_exclusive(wi, lane);
      const int Re = p0 ? we.R1 : we.R0, qe = (we.q >> p0) & 1u;
      const int Mw = qe ? wx.M1 : wx.M0;
      const unsigned hit = __ballot_sync(0xffffffffu, Mw >= 0 && b.S + Re + Mw >= TOP);
      if (hit == 0) {
        if (lane == 31) {
          sh.s = binade_value(b, b.S + (p0 ? wi.R1 : wi.R0));
          sh.i = wend;
          sh.cx = -1;
        }
      } else if (lane == __ffs(hit) - 1) {
        sh.cx = lane;
        sh.R = Re;
        sh.q = qe;
      }
    }
    __syncthreads();
    const int cw = sh.cx;
    if (cw >= 0) {
      if (warp == cw) {
        const int Rw = sh.R, qw = sh.q;
        const Xf ex = xf_exclusive(incl, lane);
        const int R = Rw + (qw ? ex.R1 : ex.R0), q = (ex.q >> qw) & 1u;
        const int M = q ? tx.M1 : tx.M0;
        const unsigned h2 = __ballot_sync(0xffffffffu, M >= 0 && b.S + R + M >= TOP);
        if (lane == __ffs(h2) - 1) {
          float sn = s;
          int in = n;
          cross_element(v, lo, hi, n, b, R, q, sn, in);
          sh.s = sn;
          sh.i = in;
        }
      }
      __syncthreads();
    }
    s = sh.s;
    i = sh.i;
    __syncthreads();  // sh is free
  }
  __syncthreads();
  if (tid == 0) {
    sh.s = s;
    sh.i = i;
  }
  __syncthreads();
}

// One CTA: the whole sum.
__global__ void __launch_bounds__(ES_T) k_exact_sum_solo(const float *v, int n, float *out) {
  __shared__ EsShared sh;
  es_solo(v, n, n, ((unsigned long long)v & 15ull) == 0, sh);
  if (threadIdx.x == 0) *out = sh.s;
}

struct EsArgs {
  const float *v;
  int n;
  float *out;
  int *comp;                // [2][ES_MAXG][8] the CTAs' composites, by step parity
  unsigned *bar;            // the barrier counter; zero before the launch, as pub
  unsigned long long *pub;  // [2] the published state: (s, tag), (i, tag), tag = step + 1
  int *err;
  unsigned long long wait_ns;  // limit of every wait
  bool hold;                   // the first state is not published (test hook)
};

// A state published by one CTA to all (each 8-byte word carries its tag).
__device__ __forceinline__ void es_publish(const EsArgs &A, float s, int i, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(A.pub),
               "l"((unsigned long long)__float_as_uint(s) | ((unsigned long long)tag << 32))
               : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(A.pub + 1),
               "l"((unsigned long long)(unsigned)i | ((unsigned long long)tag << 32))
               : "memory");
}
// Bounded wait for the state with this tag (thread 0 polls); false in every
// thread when it ran out.
__device__ __forceinline__ bool es_receive(const EsArgs &A, unsigned tag, EsShared &sh) {
  int bad = 0;
  if (threadIdx.x == 0) {
    unsigned long long a, b, t0 = 0;
    for (unsigned n = 1;; ++n) {
      asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(A.pub) : "memory");
      asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(A.pub + 1) : "memory");
      if ((unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag) break;
      if ((n & 15u) == 0 && ld_relaxed_gpu((const unsigned *)A.err) != 0) {
        bad = 1;
        break;
      }
      if ((n & 63u) == 0) {
        const unsigned long long t = gtimer();
        if (t0 == 0)
          t0 = t;
        else if (t - t0 > A.wait_ns)
          atomicOr(A.err, 2);
      }
    }
    sh.s = __uint_as_float((unsigned)a);
    sh.i = (int)(unsigned)b;
  }
  return __syncthreads_or(bad) == 0;
}

// One CTA per SM.  Step k: every CTA's chunk composite, barrier, every CTA
// walks the composites (warp 0, a scan); without a crossing all know the next
// state, otherwise the crossing CTA finds the element and publishes it.
__global__ void __launch_bounds__(ES_T) k_exact_sum(EsArgs A) {
  const int G = gridDim.x, c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = A.n;
  const bool aligned = ((unsigned long long)A.v & 15ull) == 0;
  GridBarrier bar(A.bar, (unsigned)G, A.err, A.wait_ns);
  __shared__ EsShared sh;
  unsigned tag = 1;
  if (c == 0) {
    es_solo(A.v, n, ES_SOLO, aligned, sh);
    if (tid == 0 && !A.hold) es_publish(A, sh.s, sh.i, tag);
  }
  if (!es_receive(A, tag, sh)) return;
  float s = sh.s;
  int i = sh.i;
  __syncthreads();
  for (unsigned step = 0; i < n; ++step) {
    if (step >= MAX_SEGMENTS) {
      // finish in plain sequence, still exact
      if (c == 0)
        for (; i < n; i += ES_SEQ) s = seq_block(A.v, i, min(n - i, ES_SEQ), s, sh.buf);
      break;
    }
    ++tag;
    const Binade b = binade_of(s);
    const int p0 = b.S & 1;
    const int wend = (int)min((long long)n, 2ll * (long long)i);
    int lo, hi;
    thread_range(i, wend, c, G, lo, hi);
    const Xf tx = xf_range(A.v, lo, hi, aligned, b);
    const Xf incl = xf_scan(tx, lane);
    if (lane == 31) sh.w[warp] = incl;
    __syncthreads();
    int *comp = A.comp + (size_t)(step & 1u) * ES_MAXG * 8;
    Xf wx, we;  // every warp: the warps' composites and the ones before them
    {
      wx = sh.w[lane];
      const Xf wi = xf_scan(wx, lane);
      we = xf_exclusive(wi, lane);
      if (warp == 0 && lane == 31) {
        *(int4 *)(comp + 8 * c) = make_int4(wi.R0, wi.R1, wi.M0, wi.M1);
        comp[8 * c + 4] = (int)wi.q;
      }
    }
    if (!bar.sync()) return;
    if (warp == 0) {
      // lane: the composites of chunks per * lane .. + per - 1
      const int per = (G + 31) / 32;
      Xf cx[ES_MAXG / 32];
      Xf x = xf_identity();
#pragma unroll
      for (int j = 0; j < ES_MAXG / 32; ++j) {
        const int cc = per * lane + j;
        cx[j] = xf_identity();
        if (j < per && cc < G) {
          const int4 a = __ldcg((const int4 *)(comp + 8 * cc));
          cx[j] = Xf{a.x, a.y, a.z, a.w, (unsigned)__ldcg(comp + 8 * cc + 4)};
        }
        x = xf_then(x, cx[j]);
      }
      const Xf xi = xf_scan(x, lane), xe = xf_exclusive(xi, lane);
      const int Re = p0 ? xe.R1 : xe.R0, qe = (xe.q >> p0) & 1u;
      const int M = qe ? x.M1 : x.M0;
      const unsigned hit = __ballot_sync(0xffffffffu, M >= 0 && b.S + Re + M >= TOP);
      if (hit == 0) {
        if (lane == 31) {
          sh.cx = -1;
          sh.R = p0 ? xi.R1 : xi.R0;
        }
      } else if (lane == __ffs(hit) - 1) {
        int R = Re, q = qe, at = -1;
#pragma unroll
        for (int j = 0; j < ES_MAXG / 32; ++j) {
          const int Mj = q ? cx[j].M1 : cx[j].M0;
          if (at < 0) {
            if (Mj >= 0 && b.S + R + Mj >= TOP) {
              at = per * lane + j;
            } else {
              R += q ? cx[j].R1 : cx[j].R0;
              q = (cx[j].q >> q) & 1u;
            }
          }
        }
        sh.cx = at;
        sh.R = R;
        sh.q = q;
      }
    }
    __syncthreads();
    if (sh.cx < 0) {
      s = binade_value(b, b.S + sh.R);
      i = wend;
      __syncthreads();
      continue;
    }
    if (sh.cx == c) {
      const int R0 = sh.R, q0 = sh.q;
      // the first warp of the chunk that crosses, its first thread, the element
      const int Re = R0 + (q0 ? we.R1 : we.R0), qe = (we.q >> q0) & 1u;
      const int Mw = qe ? wx.M1 : wx.M0;
      const unsigned hit = __ballot_sync(0xffffffffu, Mw >= 0 && b.S + Re + Mw >= TOP);
      const int cw = __ffs(hit) - 1;
      const int Rw = __shfl_sync(0xffffffffu, Re, cw), qw = __shfl_sync(0xffffffffu, qe, cw);
      if (warp == cw) {
        const Xf ex = xf_exclusive(incl, lane);
        const int R = Rw + (qw ? ex.R1 : ex.R0), q = (ex.q >> qw) & 1u;
        const int M = q ? tx.M1 : tx.M0;
        const unsigned h2 = __ballot_sync(0xffffffffu, M >= 0 && b.S + R + M >= TOP);
        if (lane == __ffs(h2) - 1) {
          float sn = s;
          int in = n;
          cross_element(A.v, lo, hi, n, b, R, q, sn, in);
          es_publish(A, sn, in, tag);
        }
      }
    }
    if (!es_receive(A, tag, sh)) return;
    s = sh.s;
    i = sh.i;
    __syncthreads();
  }
  if (c == 0 && tid == 0) *A.out = s;
}

}  // namespace

int exact_sum_max_grid(int device) {
  int nsm = 0, per = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_exact_sum, ES_T, 0);
  const int g = per < 1 ? 1 : nsm;
  return g < ES_MAXG ? g : ES_MAXG;
}

size_t exact_sum_comp_ints() { return 2 * (size_t)ES_MAXG * 8; }

bool exact_sum_is_cooperative(int n) { return n > ES_SOLO; }

void launch_exact_sum(const float *v, int n, float *out, const ExactSumWork &W, cudaStream_t s) {
  if (!exact_sum_is_cooperative(n)) {
    k_exact_sum_solo<<<1, ES_T, 0, s>>>(v, n, out);
    return;
  }
  EsArgs A;
  A.v = v;
  A.n = n;
  A.out = out;
  A.comp = W.comp;
  A.bar = W.bar;
  A.pub = (unsigned long long *)(W.bar + 2);
  A.err = W.err;
  A.wait_ns = W.wait_ns ? W.wait_ns : BAR_TIMEOUT_NS;
  A.hold = W.hold;
  RPBA_CUDA_CHECK(cudaMemsetAsync(W.bar, 0, ES_BAR_WORDS * sizeof(unsigned), s));
  void *args[] = {&A};
  RPBA_CUDA_CHECK(
      cudaLaunchCooperativeKernel((const void *)k_exact_sum, dim3(W.max_grid), dim3(ES_T), args, 0, s));
}

}  // namespace rpba

// ---------------------------------------------------------------------------
// Allocation-free variant of the exact float sum.
//
// Some callers cannot let a library call cudaMalloc or cudaFree: a host
// application that hands all device memory out of its own fixed-budget pool
// (a stray cudaMalloc breaks its accounting or fails when the pool owns the
// whole device), or a latency-critical loop that cannot absorb the
// device-wide synchronisation cudaFree implies.  For them this entry point
// keeps its scratch -- the CTAs' composites, the published state and the
// grid-barrier counter of k_exact_sum -- in one statically sized device
// array that every GPU loading the library holds until the process exits
// (about 16 KB).  Its size caps the grid at ES_MAXG CTAs; inputs up to
// NA_MAX_N elements are accepted on any device.
using namespace rpba;

namespace {

constexpr long long NA_MAX_N = 4194304;  // a fixed limit of the entry point
constexpr size_t NA_OFF_BAR = 2 * (size_t)ES_MAXG * 8 * sizeof(int);  // after the composites
constexpr size_t NA_OFF_ERR = NA_OFF_BAR + ES_BAR_WORDS * sizeof(unsigned);
constexpr size_t NA_BYTES = NA_OFF_ERR + 16;

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

// The array's device address belongs to the context the module was loaded
// in: after cudaDeviceReset (or when the caller makes another context
// current) it is looked up again.  Contexts are told apart by their
// process-unique id (cuCtxGetId); the two driver calls are fetched through
// the runtime, so the library does not link the driver library.
typedef CUresult (*PfnCtxGetCurrent)(CUcontext *);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long *);

constexpr int NA_MAX_DEVICES = 64;
struct NaSlot {
  unsigned long long ctx_id;  // 0: not looked up yet
  unsigned char *addr;        // device address of the scratch in that context
};
std::mutex g_na_mutex;
NaSlot g_na[NA_MAX_DEVICES];
PfnCtxGetCurrent g_ctx_current = nullptr;
PfnCtxGetId g_ctx_id = nullptr;

// Id of the calling thread's current context; 0 when none is current.
// Call with g_na_mutex held.
bool current_ctx_id(unsigned long long *id) {
  if (!g_ctx_current || !g_ctx_id) {
    void *a = nullptr, *b = nullptr;
    cudaDriverEntryPointQueryResult qa, qb;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) != cudaSuccess ||
        qa != cudaDriverEntryPointSuccess || !a ||
        cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) != cudaSuccess ||
        qb != cudaDriverEntryPointSuccess || !b)
      return false;
    g_ctx_current = (PfnCtxGetCurrent)a;
    g_ctx_id = (PfnCtxGetId)b;
  }
  CUcontext ctx = nullptr;
  if (g_ctx_current(&ctx) != CUDA_SUCCESS) return false;
  *id = 0;
  return !ctx || g_ctx_id(ctx, id) == CUDA_SUCCESS;
}

}  // namespace

extern "C" int32_t rpba_float_sequential_sum_noalloc(const float *d_v, int64_t n, float *d_out, void *stream) {
  if (!d_out || n < 0 || (n > 0 && !d_v)) return RPBA_ERR_ARG;
  if (n > NA_MAX_N) return RPBA_ERR_TOO_LARGE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RPBA_ERR_NO_DEVICE;
  if (dev < 0 || dev >= NA_MAX_DEVICES) return RPBA_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char *base;
  {
    // set-up, once per device and context, with that device current: the
    // array's name is only a host-side stand-in, so its device address is
    // looked up (the lookup also makes the runtime's context current when
    // this thread has none yet)
    std::lock_guard<std::mutex> lock(g_na_mutex);
    unsigned long long id = 0;
    if (!current_ctx_id(&id)) return RPBA_ERR_CUDA;
    if (id == 0 || g_na[dev].ctx_id != id) {
      void *p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return RPBA_ERR_CUDA;
      if (id == 0 && (!current_ctx_id(&id) || id == 0)) return RPBA_ERR_CUDA;
      g_na[dev].ctx_id = id;
      g_na[dev].addr = (unsigned char *)p;
    }
    base = g_na[dev].addr;
  }
  const int ni = (int)n;
  // until the sum is written, *d_out holds a NaN (all bits set): a grid
  // barrier that runs out leaves it there
  if (cudaMemsetAsync(d_out, 0xff, sizeof(float), s) != cudaSuccess) return RPBA_ERR_CUDA;
  if (!exact_sum_is_cooperative(ni)) {
    void *wargs[] = {(void *)&d_v, (void *)&ni, (void *)&d_out};
    return cudaLaunchKernel((const void *)k_exact_sum_solo, dim3(1), dim3(ES_T), wargs, 0, s) == cudaSuccess
               ? RPBA_OK
               : RPBA_ERR_CUDA;
  }
  int nsm = 0, per = 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_exact_sum, ES_T, 0) != cudaSuccess || nsm * per < 1)
    return RPBA_ERR_CUDA;
  // every CTA must be resident (cooperative launch) and own a slot of the array
  const int G = nsm < ES_MAXG ? nsm : ES_MAXG;
  EsArgs A;
  A.v = d_v;
  A.n = ni;
  A.out = d_out;
  A.comp = (int *)base;
  A.bar = (unsigned *)(base + NA_OFF_BAR);
  A.pub = (unsigned long long *)(A.bar + 2);
  A.err = (int *)(base + NA_OFF_ERR);
  A.wait_ns = BAR_TIMEOUT_NS;
  A.hold = false;
  // the array keeps the previous call's contents: the barrier counter, the
  // published state and the error word must start at zero; the rest is
  // written before it is read
  if (cudaMemsetAsync(A.bar, 0, NA_BYTES - NA_OFF_BAR, s) != cudaSuccess) return RPBA_ERR_CUDA;
  void *args[] = {&A};
  if (cudaLaunchCooperativeKernel((const void *)k_exact_sum, dim3(G), dim3(ES_T), args, 0, s) != cudaSuccess)
    return RPBA_ERR_CUDA;
  return RPBA_OK;
}
