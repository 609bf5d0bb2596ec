// FP32 building blocks shared by the backprojectors: packed pairs, floors without conversions, and
// divisions by values whose reciprocal is at hand.
#pragma once

#include <cuda_runtime.h>

namespace lct {

// Blackwell's packed FP32 pairs (FFMA2, FADD2, FMUL2): one instruction for two lanes, each lane
// rounded exactly as the scalar operation; x - y is written fma(y, -1, x), one rounding like the
// subtraction.
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 f2sub(float2 x, float2 y) {
  return __ffma2_rn(y, make_float2(-1.0f, -1.0f), x);
}

// Floor without conversions: for |x| < 2^22, x + 1.5 * 2^23 rounded toward -inf is
// 1.5 * 2^23 + floor(x) exactly, so its bit pattern is kFloorBits + floor(x) and subtracting the
// constant back (exact: both operands lie within a factor of two) gives floor(x).  Outside that
// range the bit pattern still orders like x, so a clamp on it clamps floor(x).
constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kFloorBits = 0x4B400000;
// the same for the 1/256 grid of 8-bit weights, |x| < 2^14, and half a step of it
constexpr float kFloorMagic8 = 49152.0f;  // 1.5 * 2^15
constexpr float kHalfStep8 = 1.0f / 512.0f;

// The hardware's approximate reciprocal and reciprocal square root without the scaling that the
// general forms wrap around them for subnormal and huge arguments (distances and row differences are
// neither); the same values otherwise.
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_fast(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// x / d rounded to nearest where r = RN(1 / d) is at hand (a constant of the launch, or one per view): the
// quotient estimate's remainder is exact in an FMA and one more FMA rounds correctly (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. R&D 34(1), 1990), except that
// a divisor whose fraction bits are all ones may leave a power of two one ulp off; 3 operations where a
// division by a variable is a subroutine.  For normal numbers: d = 0 and an infinite quotient give NaN.
// tests/test_div_by_kernel.py compiles these functions and compares every fraction of x, constant divisors and
// varying ones, with the division.
__device__ __forceinline__ float div_by(float x, float d, float r) {
  const float q = __fmul_rn(x, r);
  return fmaf(fmaf(-q, d, x), r, q);
}
__device__ __forceinline__ float2 div_by2(float2 x, float d, float r) {
  const float2 q = __fmul2_rn(x, f2(r));
  return __ffma2_rn(__ffma2_rn(q, f2(-d), x), f2(r), q);
}

}  // namespace lct
