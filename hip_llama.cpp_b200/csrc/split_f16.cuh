// fp32 values as two fp16: v times a power of two that a whole row shares = hi + lo 2^-11, hi = fp16(v), lo = fp16((v - hi) 2^11).  What fp32 prompts' products
// (gemm_f16x3.cu) and attention (attn_prefill_x3.cu) multiply.
//
// The scheme is Ootomo and Yokota's ("Recovering single precision accuracy from Tensor Cores while surpassing the FP32 theoretical peak
// performance", 2022).  A normal fp16 has 11 bits of significand, so hi and lo hold 22.  Their factor of 2^11 on lo keeps it normal down to where hi ends: without it lo
// lost its last bits from 2^-3 downwards (fp16 ends at 2^-24), now from 2^-14: a value 2^28 below the largest of a row that is brought to [2^14, 2^15) still has its 22 bits, and
// nothing is off by more than 2^-36.  A sum of products is hi.hi + 2^-11 (hi.lo + lo.hi); lo.lo, 2^-22 of a product at most, is left out.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace tha {

constexpr int SPLIT_LO = 11;
constexpr float SPLIT_UP = 2048.0f, SPLIT_DOWN = 1.0f / 2048.0f;

// two fp32 operations in one instruction
__device__ __forceinline__ float2 f32x2_mul(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f32x2_fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ uint32_t f16x2_of(float2 v) {   // v.x in the low half, nearest even, infinity beyond the range
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  return r;
}
// v times s, a power of two, split
__device__ __forceinline__ void split_f16x2(float2 v, float s, uint32_t& hi, uint32_t& lo) {
  hi = f16x2_of(f32x2_mul(v, make_float2(s, s)));
  const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  const float up = s * SPLIT_UP;
  lo = f16x2_of(f32x2_fma(h, make_float2(-SPLIT_UP, -SPLIT_UP), f32x2_mul(v, make_float2(up, up))));   // every step of it is exact but the last rounding
}
// (row kernels, bound by memory: single operations leave them more registers for loads in flight)
__device__ __forceinline__ void split_f16x4(float4 v, float s, uint2& hi, uint2& lo) {
  v.x *= s; v.y *= s; v.z *= s; v.w *= s;
  hi = make_uint2(f16x2_of(make_float2(v.x, v.y)), f16x2_of(make_float2(v.z, v.w)));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&hi.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&hi.y));
  lo = make_uint2(f16x2_of(make_float2((v.x - a.x) * SPLIT_UP, (v.y - a.y) * SPLIT_UP)), f16x2_of(make_float2((v.z - b.x) * SPLIT_UP, (v.w - b.y) * SPLIT_UP)));
}
// The power of two, 2^MOST at most, that brings |v| to [2^e, 2^(e+1)), and its inverse
template <int MOST>
__device__ __forceinline__ float split_scale(float v, int e, float* inverse) {
  static_assert(MOST <= 115, "with 2^11 on top it is a finite number, and its inverse a normal one");
  const int s = min(254 + e - (int)(__float_as_uint(v) >> 23), 127 + MOST);
  *inverse = __uint_as_float((uint32_t)(254 - s) << 23);
  return __uint_as_float((uint32_t)s << 23);
}

}  // namespace tha
