// Activations of feed-forwards, shared by the row kernels and the experts' projections.
#pragma once
#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace {

// y / d for d >= 1, without the branch of the compiler's division, so that a thread works on many quotients at once: the one from an approximate reciprocal (of d / 2^8, whose reciprocal
// is never too small), corrected once by its remainder (P. Markstein, Computation of elementary functions on the IBM RISC System/6000, 1990).  An infinite y or d leaves no remainder to
// correct by (and a zero comes out positive).  z / (1 + expf(-z)) for 2^25 numbers of N(0, 0.3^2) to N(0, 30^2): not a bit differs; nor does it below, down to fp32's smallest numbers, where y itself is never scaled.  (The
// remainder of a y below 2^-100 may be rounded off, which is an ulp of the quotient at most.)  The experts' epilogue, 128 SiLUs a thread and tile, was bound by that branch: 2048 rows of 2048
// channels, 16 experts, up projection 95 -> 73 us, of 1024 channels 60 -> 26.
__device__ __forceinline__ float over(float y, float d) {
  constexpr float S = 0.00390625f;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d * S));
  r *= S;
  const float q = y * r, better = fmaf(fmaf(-q, d, y), r, q);
  return better == better ? better : q;
}

__device__ __forceinline__ float act_apply(float z, int act) {
  switch (act) {
    case LIA_ACT_RELU: return fmaxf(z, 0.f);
    case LIA_ACT_SILU: return over(z, 1.0f + expf(-z));
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
    return over(g, 1.0f + expf(-p1 * g)) * (u + 1.0f);
  }
  return act_apply(g, act) * u;
}

// use(std::integral_constant<int, act>): the activation chosen once for a block of numbers
template <typename F> __device__ __forceinline__ void act_chosen(int act, F use) {
  switch (act) {
    case LIA_ACT_RELU: return use(std::integral_constant<int, LIA_ACT_RELU>());
    case LIA_ACT_SILU: return use(std::integral_constant<int, LIA_ACT_SILU>());
    case LIA_ACT_GELU_ERF: return use(std::integral_constant<int, LIA_ACT_GELU_ERF>());
    case LIA_ACT_GELU_TANH: return use(std::integral_constant<int, LIA_ACT_GELU_TANH>());
    case LIA_ACT_RELU_SQUARED: return use(std::integral_constant<int, LIA_ACT_RELU_SQUARED>());
    default: return use(std::integral_constant<int, LIA_ACT_NONE>());
  }
}

}  // namespace
