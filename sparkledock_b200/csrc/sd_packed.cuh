// Two FP32 values in a 64-bit register and the packed instructions of sm_100 on them: each element is
// rounded as by the scalar instruction.
#pragma once

namespace sd {

typedef unsigned long long float2x;
__device__ __forceinline__ float2x pack2(float a, float b) {
  float2x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(float2x v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ float2x add2(float2x a, float2x b) {
  float2x r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float2x mul2(float2x a, float2x b) {
  float2x r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float2x fma2(float2x a, float2x b, float2x c) {
  float2x r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

}  // namespace sd
