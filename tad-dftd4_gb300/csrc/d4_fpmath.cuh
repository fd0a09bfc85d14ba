// FP64 reciprocal and inverse square root for arguments that are positive and
// normal, without the special cases of the library functions: the PTX
// approximation (20 bits and more) and one third-order step, whose error is
// below the rounding of its last FMA.  The FP64 pipe takes 64 cycles per warp
// instruction, so the instructions saved (4 of 9 or more) are time saved.
#pragma once

#include <cuda_runtime.h>

namespace d4 {

// y (1 + e + e^2), e = 1 - d y (Householder's method for 1 / d); d beyond
// 2^1022 gives 0.
__device__ __forceinline__ double rcp_pos(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// y (1 + e / 2 + 3 e^2 / 8), e = 1 - d y^2 (the binomial series of
// (1 - e)^(-1/2)).
__device__ __forceinline__ double rsqrt_pos(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-(d * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

}  // namespace d4
