// group_barrier.cuh -- the barrier of the CTAs that step a lattice together inside one launch.
//
// Only cooperative launches use it: all their CTAs are resident, so they always run together.  Every
// wait is bounded.
#pragma once
#include <cuda_runtime.h>

#include "lbm_step_tma.cuh"

namespace hlbm {

constexpr int GROUP_ERR_TIMEOUT = 2;

// All CTAs of the launch have finished their step: one arrival per CTA on `counter`, and a bounded wait
// for it to reach `target` (arrivals since the launch began).  False when the wait ran out (uniform
// over the CTA).  Measured alone on 148 CTAs: 1.2 us.  A release word apart from the counter takes
// 0.2 us more, two levels (cluster, then counter) 0.5 us more, and a word per CTA that every CTA
// polls 2 to 5 us more.
__device__ __forceinline__ bool group_barrier(unsigned* counter, unsigned target, long long limit, int* err, int* bail) {
  __syncthreads();
  if (threadIdx.x == 0) {
    // release: the CTA's stores, ordered before by the barrier, are visible to who sees the arrival
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    unsigned long long t0 = 0;
    for (long long polls = 1;; polls++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) break;
      bool out = polls >= limit;
      if ((polls & 1023) == 0) {
        const unsigned long long t = global_ns();
        if (t0 == 0) t0 = t;
        out = out || t - t0 > MBAR_WAIT_NS;
      }
      if (out) {
        atomicExch(err, GROUP_ERR_TIMEOUT);
        *bail = 1;
        break;
      }
    }
  }
  __syncthreads();
  return *bail == 0;
}

// The end of a launch, called by every thread: the last CTA to leave (every other one has passed, or
// given up, its barriers) clears both counters for the next launch.
__device__ __forceinline__ void group_leave(unsigned* left, unsigned* counter) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(left, 1u) == gridDim.x - 1) {
      *counter = 0;
      *left = 0;
    }
  }
}

}  // namespace hlbm
