// f32x2.cuh -- packed pairs of floats (the .f32x2 instructions of sm_100 and
// later: two IEEE operations, round to nearest, the bits of two scalar ones)
// and three-operand minimum and maximum.
#pragma once
#include <cuda_runtime.h>

namespace tsim {

// min / max of three floats in one instruction (exact, like two fminf /
// fmaxf: a NaN operand is ignored)
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

union PackedF2 {
  float2 f;
  unsigned long long u;
};
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  PackedF2 x{a}, y{b}, r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(x.u), "l"(y.u));
  return r.f;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  PackedF2 x{a}, y{b}, r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(x.u), "l"(y.u));
  return r.f;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  PackedF2 x{a}, y{b}, z{c}, r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(x.u), "l"(y.u), "l"(z.u));
  return r.f;
}

}  // namespace tsim
