// Barrier of the CTAs of a cooperative launch, with a bounded wait.
#pragma once

#include "d4_common.cuh"
#include "d4_tc.cuh"

namespace d4 {

// One arrival per CTA on a counter that only grows; target = CTAs x barriers
// passed.  False when ``limit_ns`` of the global timer ran out (the status word then
// reports it and every CTA leaves, each after its own wait at most); ``dead`` is the
// CTA's shared flag, cleared at its start.
__device__ __forceinline__ bool group_barrier(unsigned *counter, unsigned target, int &dead,
                                              int *status,
                                              unsigned long long limit_ns = tc::WAIT_LIMIT_NS) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    unsigned v = 0;
    unsigned long long t0 = 0;
    for (unsigned k = 0;; ++k) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= target) break;
      if ((k & 63u) == 63u) {  // (the timer is not read while a barrier takes its usual time)
        const unsigned long long now = tc::global_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > limit_ns) break;
      }
    }
    if (v < target) {
      set_status(status, D4_ERR_DEVICE_TIMEOUT);
      dead = 1;
    }
  }
  __syncthreads();
  return dead == 0;
}

// Whether an earlier launch of the call gave up on such a wait: the rest of the
// call's solves leave at once (its results are incomplete, as the status says).
__device__ __forceinline__ bool group_gave_up(const int *status) {
  return *(const volatile int *)status == D4_ERR_DEVICE_TIMEOUT;
}

}  // namespace d4
