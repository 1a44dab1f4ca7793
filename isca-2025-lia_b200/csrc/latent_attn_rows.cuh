// What the kernels of latent portions over expanded keys and values share (latent_attn_mma.cu: mma.sync; latent_attn_sm100.cu: tcgen05): their arguments, the row that is formed again on the CUDA cores.
#pragma once
#include <math.h>

#include "mma.cuh"

constexpr int MAX_PORTIONS = 16;        // of one launch

struct Portion {
  const bf16* kr;       // the shared rotated key part of the first latent it sees
  int row0, n, pos0;    // its rows, and the position of the first among the latents it sees
  int part0, tile0;     // its first expanded row and its first tile of rows
};

struct ExpandedArgs {
  const bf16* q;        // rows of H heads of DN + DR channels, the first DN unrotated
  const float* qr;      // [row][H][qr_stride]: the rotated DR channels
  const bf16* parts;    // [latent][2 nh][3][DN]: keys of the heads h0 .. h0 + nh - 1, then values
  const float* gate;    // [row][H] or null
  const float* sink;    // [H] or null
  void* out;            // [row][H * DN]
  long long kr_stride;
  int ldq, qr_stride, H, h0, nh, window, out_f32, np;
  float scale;
  Portion p[MAX_PORTIONS];
};

namespace {

// One row and head over the latents [lo, hi] by one warp on the CUDA cores: lane j scores every 32nd key, lane l owns the value columns l, l + 32, ...
template <int DN> struct PlainRow {
  float m, l, o[DN / 32];
};
template <int DN, int DR>
__device__ __noinline__ PlainRow<DN> plain_row(const bf16* q, const float* qr, const bf16* keys, const bf16* vals, size_t stride, const bf16* key_rot, long long rot_stride, int lo,
                                               int hi, float scale) {
  const int lane = threadIdx.x & 31;
  auto whole = [](const bf16* p) { return __bfloat162float(p[0]) + (__bfloat162float(p[DN]) + __bfloat162float(p[2 * DN])); };
  PlainRow<DN> y;
  y.m = -INFINITY;
  y.l = 0.f;
#pragma unroll
  for (int c = 0; c < DN / 32; ++c) y.o[c] = 0.f;
  for (int j0 = lo; j0 <= hi; j0 += 32) {
    const int nk = min(32, hi + 1 - j0);
    float s = -INFINITY;
    if (lane < nk) {
      float part[8] = {};                                          // eight short chains
      for (int d = 0; d < DN; d += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) part[k] = fmaf(__bfloat162float(q[d + k]), whole(keys + (size_t)(j0 + lane) * stride + d + k), part[k]);
      for (int d = 0; d < DR; d += 8)
#pragma unroll
        for (int k = 0; k < 8; ++k) part[k] = fmaf(qr[d + k], __bfloat162float(key_rot[(size_t)(j0 + lane) * rot_stride + d + k]), part[k]);
      s = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
      s *= scale;
    }
    const float m = fmaxf(y.m, warp_max(s)), base = m == -INFINITY ? 0.f : m, p = expf(s - base), al = expf(y.m - base);
    y.m = m;
    y.l = fmaf(y.l, al, warp_sum(p));
#pragma unroll
    for (int c = 0; c < DN / 32; ++c) y.o[c] *= al;
    for (int j = 0; j < nk; ++j) {
      const float w = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
      for (int c = 0; c < DN / 32; ++c) y.o[c] = fmaf(w, whole(vals + (size_t)(j0 + j) * stride + lane + 32 * c), y.o[c]);
    }
  }
  return y;
}

}  // namespace
