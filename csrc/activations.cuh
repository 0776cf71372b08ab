// Activations of the GEMM epilogues (gemm_tc.cu, gemm_wide.cu).
#pragma once
#include <cuda_runtime.h>

namespace b2b {
namespace {

__device__ __forceinline__ float relu_sq(float x) { const float r = fmaxf(x, 0.f); return r * r; }
// xIELU: z > 0: ap z^2 + z/2;  z <= 0: an (e^z - 1 - z) + z/2
__device__ __forceinline__ float xielu(float x, float ap, float an) {
  return x > 0.f ? ap * x * x + 0.5f * x : an * (expm1f(x) - x) + 0.5f * x;
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  return 0.5f * x * (1.f + tanhf(u));
}
__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }

}  // namespace
}  // namespace b2b
