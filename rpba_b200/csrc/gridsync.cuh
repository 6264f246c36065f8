// gridsync.cuh -- bounded grid-wide barriers for cooperative launches.
#pragma once

#include <cuda_runtime.h>

namespace rpba {

constexpr unsigned long long BAR_TIMEOUT_NS = 2000000000ull;  // 2 s

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void red_add_gpu(unsigned *p, unsigned v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed_gpu(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier over all CTAs of a cooperative launch (co-residency guaranteed).
// *cnt counts arrivals over the whole launch (zero before it); barrier number
// e is passed once it reaches e x nblocks, so a CTA's arrival is one
// fire-and-forget reduction and the wait one polled word: no generation to
// read first, nothing to reset.  The wait is bounded: after limit_ns it sets
// bit 2 of *err; once *err is set every waiting CTA gives up, sync() returns
// false in all its threads and the caller leaves the kernel.  The clock is
// read every 64 polls only (a poll is an L2 round trip).
// Measured: 1.4 us less a barrier than arriving with a returning atomic, a
// generation word, a sleeping poll and every thread reading the error word
// (FP64 PCG of 3,000 cameras, 2,852 iterations of two barriers over 148 CTAs:
// 69.6 -> 61.6 ms).
struct GridBarrier {
  unsigned *cnt;
  unsigned nblocks;
  int *err;
  unsigned long long limit_ns;
  unsigned target;  // used by thread 0

  __device__ __forceinline__ GridBarrier(unsigned *cnt_, unsigned nblocks_, int *err_,
                                         unsigned long long limit_ns_ = BAR_TIMEOUT_NS)
      : cnt(cnt_), nblocks(nblocks_), err(err_), limit_ns(limit_ns_), target(0) {}

  // Arrival without the wait, for a CTA that needs none of the others'
  // results yet (it must not call sync() on the same barrier).
  __device__ __forceinline__ void arrive() {
    __syncthreads();
    if (threadIdx.x == 0) {
      fence_gpu();
      red_add_gpu(cnt, 1u);
    }
  }

  __device__ __forceinline__ bool sync() {
    __syncthreads();
    int bad = 0;
    if (threadIdx.x == 0) {
      target += nblocks;
      fence_gpu();
      red_add_gpu(cnt, 1u);
      unsigned long long t0 = 0;
      for (unsigned n = 1;; ++n) {
        const unsigned e = ld_relaxed_gpu((const unsigned *)err);
        const unsigned v = ld_relaxed_gpu(cnt);
        bad = e != 0;
        if (bad || (int)(v - target) >= 0) break;
        if ((n & 63u) == 0) {
          const unsigned long long t = gtimer();
          if (t0 == 0)
            t0 = t;
          else if (t - t0 > limit_ns)
            atomicOr(err, 2);
        }
      }
      fence_gpu();
    }
    return __syncthreads_or(bad) == 0;
  }
};

}  // namespace rpba
