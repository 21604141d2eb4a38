// Activations of the gated linear units, shared by the sequence operators and the products that end in one (the same bits from either).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace kb2act {

__device__ __forceinline__ float gelu_tanh(float z) {
  return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
// x / d for d >= 1, infinity with it, without a branch: an approximate quotient and one step along its residual (Markstein 1990, "Computation of elementary
// functions on the IBM RISC System/6000 processor").  Where the residual is not a number (d or x infinite) the product is the answer, and where it is zero the
// product stays as it is: a step of zero would make -0 a +0.  In place of x / d: the convolution of 4096 tokens x 8192
// channels 88 -> 80 us.  Errors of silu against fp64 over 4 M numbers each of five scales are those
// of the quotient: at most 2.14e-7, 3.7e-8 to 4.5e-8 in the mean.
__device__ __forceinline__ float over(float x, float d) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = x * r, left = fmaf(-q, d, x);
  return fabsf(left) > 0.f ? fmaf(left, r, q) : q;
}
__device__ __forceinline__ float silu(float z) { return over(z, 1.f + expf(-z)); }
// what a gate's number multiplies by: silu, or its sigmoid
__device__ __forceinline__ float gate_value(float z, bool sigmoid) { return over(sigmoid ? 1.f : z, 1.f + expf(-z)); }
// kind 0: gelu_tanh(g) u; 1: silu(g) u; 2: g' sigmoid(alpha g') (u' + 1) with g' = min(g, limit), u' = clamp(u, -limit, limit); 3: relu(g)^2
__device__ __forceinline__ float glu_value(float g, float u, int kind, float limit, float alpha) {
  if (kind == 3) return g > 0.f ? g * g : 0.f;
  if (kind == 0) return gelu_tanh(g) * u;
  if (kind == 1) return silu(g) * u;
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return over(g, 1.f + expf(-alpha * g)) * (u + 1.f);
}

}  // namespace kb2act
