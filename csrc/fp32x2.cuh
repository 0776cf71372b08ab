// Pairs of fp32 values in one register pair: the same IEEE results as two scalar operations at half the issue slots.
#pragma once
#include <cuda_runtime.h>

namespace b2b {
namespace {

typedef unsigned long long pair32;
__device__ __forceinline__ pair32 pack32(float lo, float hi) {
  pair32 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack32(pair32 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ pair32 add2(pair32 a, pair32 b) {
  pair32 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair32 mul2(pair32 a, pair32 b) {
  pair32 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair32 fma2(pair32 a, pair32 b, pair32 c) {
  pair32 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

}  // namespace
}  // namespace b2b
