// The activations of routed experts' products, shared by their kernels.
#pragma once

#include "common.cuh"

namespace srlm {

// limit <= 0: the plain gated form, gate * logistic(gate) * up
__device__ __forceinline__ float clamped_glu(float gate, float up, float limit, float alpha) {
  if (!(limit > 0.f)) return gate * (1.f / (1.f + expf(-gate))) * up;
  const float g = fminf(gate, limit);
  const float u = fminf(fmaxf(up, -limit), limit);
  return g * (1.f / (1.f + expf(-alpha * g))) * (u + 1.f);
}

// The activation of an expert without a gate: 0 none, 1 the exact gelu, 2 the square of the positive part.
__device__ __forceinline__ float plain_activation(float z, int act) {
  if (act == 2) return z < 0.f ? 0.f : z * z;      // (a NaN stays one)
  return act == 1 ? 0.5f * z * (1.f + erff(z * 0.70710678118654752440f)) : z;
}

}  // namespace srlm
