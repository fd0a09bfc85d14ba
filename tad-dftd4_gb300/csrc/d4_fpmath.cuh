// FP64 reciprocal and inverse square root and an FP32 exponential, without the
// special cases and instructions of the library functions that their callers do
// not need.  A warp takes the FP64 pipe for 64 cycles per instruction, so the
// instructions saved (4 of 9 or more) are time saved.
//
// Errors and edges are tested over the whole range (tests/test_gpu_fpmath.py).
#pragma once

#include <cuda_runtime.h>

#include "d4_common.cuh"

namespace d4 {

// 0, subnormal, infinite or NaN, by the exponent (not an FP64 instruction).
__device__ __forceinline__ bool fp64_edge(double y) {
  return ((__double2hiint(y) + 0x00100000) & 0x7fe00000) == 0;
}

// 1 / d for d >= 0: the PTX approximation (20 bits and more) and one third-order
// step, y (1 + e + e^2) with e = 1 - d y (Householder's method), whose error is
// below 0.01 of its last FMA's rounding (0.504 ulp measured).  d beyond 2^1022 and
// infinity give 0, 0 and subnormals infinity.  EDGE false: d is normal and below
// 2^1022.
template <bool EDGE = true>
__device__ __forceinline__ double rcp_pos(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  const double r = fma(y, fma(e, e, e), y);
  return EDGE && fp64_edge(y) ? y : r;
}

// 1 / sqrt(d) for d >= 0 likewise, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - d y^2 (the
// binomial series of (1 - e)^(-1/2)); the rounding of d y adds up to half an ulp
// (0.97 measured).
// Infinity gives 0, 0 and subnormals infinity.
template <bool EDGE = true>
__device__ __forceinline__ double rsqrt_pos(double d) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-(d * y), y, 1.0);
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  return EDGE && fp64_edge(y) ? y : r;
}

// exp(x), |x| <= 80, rounded once: reduction by ln 2 = 355/512 - 2.1e-4 (Cody and
// Waite, Software Manual for the Elementary Functions, 1980) and the series, its
// first terms in double-float: within 0.502 ulp of exp (0.501 measured), where an
// FP64 exp rounded to FP32 is within 0.5.  In place of that, whose 30 FP64
// instructions for every reference of every atom were most of the weights' time.
__device__ __forceinline__ float exp_once(dfl x) {
  const float n = rintf(x.hi * 1.44269504f);
  const float ch = 2.1219444e-4f;
  constexpr float cl = (float)(2.1219444005469058277e-4 - (double)2.1219444e-4f);
  const float p = n * ch;
  const dfl t = df_two_sum(fmaf(n, -0.693359375f, x.hi), p);  // (exact: few bits)
  const dfl r = df_fast(t.hi, t.lo + (fmaf(n, ch, -p) + fmaf(n, cl, x.lo)));
  const dfl r2 = df_mul(r, r);
  const dfl r3 = df_mul(df_mul(r2, r), dfl{1.f / 6.f, (float)(1.0 / 6.0 - (double)(1.f / 6.f))});
  const float q = fmaf(r.hi, fmaf(r.hi, fmaf(r.hi, fmaf(r.hi, fmaf(r.hi, 1.f / 362880.f,
                       1.f / 40320.f), 1.f / 5040.f), 1.f / 720.f), 1.f / 120.f), 1.f / 24.f);
  const dfl tail = df_two_sum(r3.hi, r2.hi * r2.hi * q);
  const dfl h = df_two_sum(0.5f * r2.hi, tail.hi);
  const dfl u = df_two_sum(r.hi, h.hi);
  const dfl v = df_two_sum(1.f, u.hi);
  const float lo = v.lo + (u.lo + (r.lo + (h.lo + fmaf(0.5f, r2.lo, tail.lo + r3.lo))));
  return (v.hi + lo) * __int_as_float(((int)n + 127) << 23);
}

}  // namespace d4
