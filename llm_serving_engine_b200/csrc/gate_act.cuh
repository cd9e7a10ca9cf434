// The gated feed-forwards' activations.
#pragma once
#include <cuda_runtime.h>

// ACT 0: silu(g) = g / (1 + exp(-g)).  ACT 1: gelu(g) = 0.5 g (1 + tanh(sqrt(2/pi) (g + 0.044715 g^3))).
// FAST: the result is rounded to bfloat16, far more coarsely than the fast exponential and division err.
template <int ACT, bool FAST>
__device__ __forceinline__ float gate_act(float g) {
  if (ACT == 2) return fmaxf(g, 0.f);
  if (ACT == 3) return FAST ? __fdividef(g, 1.0f + __expf(-1.702f * g)) : g / (1.0f + expf(-1.702f * g));
  if (ACT == 0) return FAST ? __fdividef(g, 1.0f + __expf(-g)) : g / (1.0f + expf(-g));
  const float inner = 0.7978845608028654f * fmaf(0.044715f * g * g, g, g);
  if (FAST) return g - __fdividef(g, 1.0f + __expf(2.0f * inner));   // 0.5 g (1 + tanh x) = g - g / (1 + exp(2x))
  return 0.5f * g * (1.0f + tanhf(inner));
}

// The product of the activated gate and the up value.  ACT 3 (clamped swish): g' = min(g, limit), u' = clamp(u, -limit,
// limit), g' sigmoid(1.702 g') (u' + 1); the others: act(g) u, `limit` not read.
template <int ACT, bool FAST>
__device__ __forceinline__ float gate_mul(float g, float u, float limit) {
  if (ACT == 3) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit) + 1.0f;
  }
  return gate_act<ACT, FAST>(g) * u;
}
