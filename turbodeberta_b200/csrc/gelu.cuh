// The exact GELU, x * Phi(x), for results in fp32 and in bf16.
#pragma once
#include <cuda_bf16.h>

namespace tdb {

// Phi(-|x|) = erfc(|x| / sqrt 2) / 2 by formula 7.1.26 of Abramowitz and Stegun's handbook (absolute error below 1.5e-7;
// relative to the value 5e-5 down to x = -3 and 2e-3 down to x = -5, where 1 + erf(x) in fp32 is off by 5e-2): for results that
// are rounded to bf16.  One path for every x, two special-function operations; erff diverges into two branches of some forty instructions.
__device__ __forceinline__ float phi_tail(float ax) {
  float t, e;                                        // 1 / (1 + 0.3275911 z) and exp(-z^2), z = ax / sqrt 2, one instruction each
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(0.3275911f * 0.70710678118654752f, ax, 1.f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(ax * ax * (-0.5f * 1.4426950408889634f)));
  // the formula's coefficients with the half folded in
  const float poly = t * fmaf(t, fmaf(t, fmaf(t, fmaf(t, 0.5307027145f, -0.7265760135f), 0.7107068705f), -0.142248368f), 0.127414796f);
  return poly * e;
}
__device__ __forceinline__ float gelu(float x, float) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu(float x, __nv_bfloat16) {
  const float tail = x * phi_tail(fabsf(x));
  return x < 0.f ? tail : x - tail;
}

}  // namespace tdb
