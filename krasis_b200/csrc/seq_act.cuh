// Activations of the gated linear units, shared by the sequence operators and the products that end in one (the same bits from either).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace kb2act {

__device__ __forceinline__ float gelu_tanh(float z) {
  return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
// kind 0: gelu_tanh(g) u; 1: silu(g) u; 2: g' sigmoid(alpha g') (u' + 1) with g' = min(g, limit), u' = clamp(u, -limit, limit); 3: relu(g)^2
__device__ __forceinline__ float glu_value(float g, float u, int kind, float limit, float alpha) {
  if (kind == 3) return g > 0.f ? g * g : 0.f;
  if (kind == 0) return gelu_tanh(g) * u;
  if (kind == 1) return silu(g) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g / (1.f + expf(-alpha * g)) * (u + 1.f);
}

}  // namespace kb2act
