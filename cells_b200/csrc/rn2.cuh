// Correctly rounded f32 reciprocal, quotient and square root of two values at once: the hardware's
// approximations, then the residual of the estimate by FMA and one correction in packed f32x2 (Newton's
// iteration as in P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990). The bits are those of 1 / x, a / b and sqrtf(x) for operands and results between
// 2^-100 and 2^100; zeros, infinities and denormals are the caller's to keep out.
#pragma once

namespace cells {

__device__ __forceinline__ float2 rn_neg2(float2 a) { return __fmul2_rn(a, make_float2(-1.0f, -1.0f)); }

// 1 / x
__device__ __forceinline__ float2 rn_rcp2(float2 x) {
  float2 y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
  return __ffma2_rn(y, __ffma2_rn(rn_neg2(x), y, make_float2(1.0f, 1.0f)), y);
}

// a / b, given y = 1 / b correctly rounded
__device__ __forceinline__ float2 rn_div2(float2 a, float2 b, float2 y) {
  const float2 q = __fmul2_rn(a, y);
  return __ffma2_rn(__ffma2_rn(rn_neg2(b), q, a), y, q);
}

// sqrt(x)
__device__ __forceinline__ float2 rn_sqrt2(float2 x) {
  float2 y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(x.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(x.y));
  const float2 g = __fmul2_rn(x, y), h = __fmul2_rn(y, make_float2(0.5f, 0.5f));
  return __ffma2_rn(__ffma2_rn(rn_neg2(g), g, x), h, g);
}

}  // namespace cells
