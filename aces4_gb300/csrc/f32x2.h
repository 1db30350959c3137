// Packed FP32 arithmetic (two values per instruction, sm_100 and later) and
// conversions of small integers that stay off the conversion pipe.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace a4g {
namespace {

typedef unsigned long long F32x2;

__device__ __forceinline__ F32x2 pack2(float lo, float hi) {
  F32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(F32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c) {
  F32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ F32x2 add2(F32x2 a, F32x2 b) {
  F32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint32_t bf16x2_of(F32x2 v) {
  float lo, hi;
  unpack2(v, lo, hi);
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// x + kRintMagic - kRintMagic rounds |x| < 2^22 to the nearest integer.
constexpr float kRintMagic = 12582912.0f;  // 1.5 2^23

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

}  // namespace
}  // namespace a4g
