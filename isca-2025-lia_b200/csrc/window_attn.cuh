// What the window-attention kernels share (window_attn.cu: CUDA cores, any type and size; window_attn_mma.cu: tensor cores, bf16
// caches): their arguments, the visible range of a position, the output gate.
#pragma once
#include <math.h>

#include "common.cuh"

struct WindowArgs {
  int H, G, dim, vdim, window;
  int HB, NG, QR, nsplit;      // query heads per block (spanning at most NG key/value heads), rows per block, key ranges per row
  float scale, softcap;
  int q_f32, gate_mode, ldg;   // queries in fp32; gate: 0 none, 1 fp32 [M][H] as is, 2 sigmoid of the activations' type [M][ldg], per channel
  int chunk = 0;               // > 0: a position sees only the keys of its own block of `chunk` positions (counted from the sequence's start)
  int v_div = 1;               // key head g reads value head g / v_div (the value cache holds G / v_div heads)
  int out_f32 = 0;             // the output in fp32 whatever the caches hold
};

// what the scores and the output take besides q, k, v (each may be null)
struct WindowExtras {
  const float* temp;     // [H] multiplies the scaled score
  const float* slopes;   // [H] slopes[h] * (pos - j) is taken off the score
  const float* sink;     // [H] exp(sink_h) joins the softmax's denominator
  const void* gate;      // see WindowArgs::gate_mode
};

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

// first position a query at `pos` sees: the window's start, and the start of its chunk if the mask is chunked
__host__ __device__ __forceinline__ int first_key(const WindowArgs& a, int pos) {
  int lo = pos - a.window + 1 > 0 ? pos - a.window + 1 : 0;
  if (a.chunk > 0 && pos - pos % a.chunk > lo) lo = pos - pos % a.chunk;
  return lo;
}

// the output in the caches' type or, `out_f32`, in fp32
template <typename T>
__device__ __forceinline__ void store_out(T* out, size_t at, float v, const WindowArgs& a) {
  if (a.out_f32) reinterpret_cast<float*>(out)[at] = v;
  else stf(out + at, v);
}

template <typename T>
__device__ __forceinline__ float gate_of(const WindowExtras& x, const WindowArgs& a, size_t row, int h, int ch) {
  if (a.gate_mode == 1) return reinterpret_cast<const float*>(x.gate)[row * a.H + h];
  if (a.gate_mode == 2) return 1.0f / (1.0f + expf(-ldf(reinterpret_cast<const T*>(x.gate) + row * a.ldg + (size_t)h * a.vdim + ch)));
  return 1.0f;
}

}  // namespace

// out[rh] = sum of the parts of (row, head) rh, see window_attn.cu
int window_combine(const float* part, const float2* part_ml, void* out, int act_f32, int M, const WindowExtras& x, const WindowArgs& a, cudaStream_t stream);
