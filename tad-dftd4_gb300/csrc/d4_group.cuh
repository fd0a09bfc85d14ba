// Barrier of the CTAs of a cooperative launch, with a bounded wait.
#pragma once

#include "d4_common.cuh"

namespace d4 {

constexpr unsigned GROUP_POLLS = 1u << 22;  // of a barrier (about two seconds)

// One arrival per CTA on a counter that only grows; target = CTAs x barriers
// passed.  False after GROUP_POLLS polls (the status word then reports it and
// every CTA leaves); ``dead`` is the CTA's shared flag, cleared at its start.
__device__ __forceinline__ bool group_barrier(unsigned *counter, unsigned target, int &dead,
                                              int *status) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    unsigned v = 0, k = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
    } while (v < target && ++k < GROUP_POLLS);
    if (v < target) {
      set_status(status, D4_ERR_DEVICE_TIMEOUT);
      dead = 1;
    }
  }
  __syncthreads();
  return dead == 0;
}

}  // namespace d4
