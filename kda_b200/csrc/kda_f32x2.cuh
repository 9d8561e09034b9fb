// Two fp32 values in one 64-bit register: sm_100 multiplies and adds a pair in one instruction.
#pragma once

#include "kda_common.cuh"

namespace kda {

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair(float x, float y) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 halves(f32x2 v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// 16 bytes of shared or global memory as two pairs
struct F4 { f32x2 a, b; };
__device__ __forceinline__ F4 lds4(const float* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void sts4(float* p, const F4& x) { *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x.a, x.b); }

}  // namespace kda
