// What the epilogues compute element by element, and moves of four floats.
#pragma once

#include "gemm.h"

namespace petb {

// 1 / (1 + exp(-x)), the reciprocal from the hardware's estimate (within 1 ulp) and one Newton-Raphson step, which leaves
// the rounding of its last fma. Relative error: expf's ulp (2^-23 at most), the sum's rounding and that one (2^-24 each), 2^-22
// in all; the quotient's is the same. The quotient compiles into a call that spends 140 clocks an element in a GEMM's
// epilogue, this into a dozen instructions that overlap. The argument is bounded so that exp stays finite; the bound passes a
// NaN on (fminf would put 88 in its place). Below x = -87.3 the estimate is no longer a normal number and the result is 0,
// where the quotient's last values are subnormal.
__device__ __forceinline__ float sigmoid_f(float x) {
  float a, r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(a) : "f"(-x), "f"(88.0f));
  const float d = 1.0f + expf(a);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return fmaf(r, fmaf(-d, r, 1.0f), r);
}
__device__ __forceinline__ float silu_f(float x) { return x * sigmoid_f(x); }
// d silu / dx = s (1 + x (1 - s))
__device__ __forceinline__ float dsilu_f(float x) {
  const float s = sigmoid_f(x);
  return s * (1.0f + x * (1.0f - s));
}

constexpr float kRmsEps = 1.1920928955078125e-07f;  // the reference's kRmsNormEps (src/ops.hpp:195)

// 1 / sqrt(x) for x > 0, from the hardware's estimate r and one Newton-Raphson step r + r (1 - x r^2) / 2, the remainder 1 - x r^2 with
// what the product x r was rounded by: within 0.51 ulp, closer than the quotient of a root, which is rounded twice. (That compiles into
// two calls, whose registers are the epilogue's.) Infinity gives 0.
__device__ __forceinline__ float reciprocal_root(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float h = x * r, rest = fmaf(-h, r, 1.f) - fmaf(x, r, -h) * r;
  return x < 1e38f ? fmaf(0.5f * r, rest, r) : r;
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

__device__ __forceinline__ float max_abs4(float a, float b, float c, float d) {
  return fmaxf(fmaxf(fabsf(a), fabsf(b)), fmaxf(fabsf(c), fabsf(d)));
}

}  // namespace petb
