// Activations of feed-forwards, shared by the row kernels and the experts' projections.
#pragma once
#include "common.cuh"

namespace {

__device__ __forceinline__ float act_apply(float z, int act) {
  switch (act) {
    case LIA_ACT_RELU: return fmaxf(z, 0.f);
    case LIA_ACT_SILU: return z / (1.0f + expf(-z));
    case LIA_ACT_GELU_ERF: return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
    case LIA_ACT_GELU_TANH: return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
    case LIA_ACT_RELU_SQUARED: return fmaxf(z, 0.f) * fmaxf(z, 0.f);
    default: return z;
  }
}

// the product of a gated feed-forward: act(g) * u, or (LIA_ACT_CLAMPED_SWISH, p0 = limit, p1 = alpha) with g' = min(g, limit) and
// u' = clamp(u, -limit, limit): g' * sigmoid(alpha g') * (u' + 1)
__device__ __forceinline__ float gated_apply(float g, float u, int act, float p0, float p1) {
  if (act == LIA_ACT_CLAMPED_SWISH) {
    g = fminf(g, p0);
    u = fminf(fmaxf(u, -p0), p0);
    return g / (1.0f + expf(-p1 * g)) * (u + 1.0f);
  }
  return act_apply(g, act) * u;
}

}  // namespace
