// Exponentials to the accuracy of the correctly rounded single-precision ones, whatever the compiler's fast-math switch makes of expf:
// __expf(x) is documented to be good to 2 + 1.173 |x| units in the last place (measured: 4.5e-7 relative where exp(A_log) is 16).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// Rounded once.  For scalars per token and head: a handful of fp64 operations each.
__device__ __forceinline__ float exp_rn(float x) { return (float)exp((double)x); }

// 1 / (1 + exp(-x)) without an exponential of its own: expm1f is one of the functions fast math leaves alone, 2 + expm1(-x) does
// not cancel (expm1 > -1) and overflows where the quotient is zero.
__device__ __forceinline__ float sigmoid_fine(float x) { return __fdiv_rn(1.f, 2.f + expm1f(-x)); }

// exp(x) for x <= 0 from the hardware's 2^t: what the product t = x log2(e) lost to rounding, r = x log2(e) - t to twice the precision,
// comes back as a factor 2^r = 1 + r ln 2.
__device__ __forceinline__ float exp_neg_fine(float x) {
  constexpr float L = 1.4426950408889634f, L_LO = 1.4426950408889634 - (double)L;
  const float t = x * L, r = fmaf(x, L_LO, fmaf(x, L, -t));
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
  return x > -88.f ? fmaf(e, r * 0.6931471805599453f, e) : e;  // (t = -inf leaves no remainder)
}
