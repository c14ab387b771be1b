// Pairs of float32 values in one register pair: Blackwell's packed FP32
// instructions (add, multiply and fused multiply-add of two values, each
// rounded to nearest) take one issue slot for two results. They run at the
// scalar instructions' result rate (measured 120 results per SM and clock
// either way), so kernels bound by the issue rate with the FMA pipe half
// idle gain from them.
#pragma once

#include <cuda_runtime.h>

namespace ss {

__device__ __forceinline__ float2 pk(float a, float b) {
  return make_float2(a, b);
}
__device__ __forceinline__ float2 pk1(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  return __fadd2_rn(a, b);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  return __fmul2_rn(a, b);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  return __ffma2_rn(a, b, c);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long x, y, z;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(z));
  return r;
}

// s + e == a + b exactly (Knuth).
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s,
                                         float2 &e) {
  s = add2(a, b);
  const float2 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

}  // namespace ss
