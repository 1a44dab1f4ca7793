// What the tensor-core forms of window attention share (window_attn_mma.cu: mma.sync; window_attn_sm100.cu: tcgen05): the scores behind their products, the row that is formed again on
// the CUDA cores, the portion that a tile of rows belongs to.
#pragma once
#include "mma.cuh"
#include "window_attn.cuh"

namespace {

// Of the prompts with heads of 128 + 128 channels, portions of up to so many rows may go to mma.sync (lia_window_prompt_form)
constexpr int SHORT_ROWS = 128;

// scores of one thread, in place: dot products * mul -> soft-capped, less the distance's cost.  dist(i) = query position - key position of score i.
// tanh of small arguments (real scores are far below the cap) is its Taylor series up to the 9th power: below 0.3 the rest is under 6e-8 of
// the value, one rounding, at a third of the instructions of tanhf, which with exp bounds this kernel as much as the products do.
template <int N, typename Dist> __device__ __forceinline__ void finish_scores(float (&s)[N], float mul, const WindowArgs& a, float slope, const Dist& dist) {
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] *= mul;
  if (a.softcap > 0.f) {
    // s / softcap as the division rounds it, without its branch: the product with the reciprocal, corrected once by its remainder (P. Markstein, Computation of elementary functions
    // on the IBM RISC System/6000, 1990); an infinite score leaves no remainder to correct by
    const float inv = 1.0f / a.softcap;
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float q = s[i] * inv, better = fmaf(fmaf(-q, a.softcap, s[i]), inv, q);
      s[i] = better == better ? better : q;
      top = fmaxf(top, fabsf(s[i]));
      if (s[i] != s[i]) top = INFINITY;
    }
    if (top <= 0.3f) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float z = s[i] * s[i];
        const float p = z * fmaf(z, fmaf(z, fmaf(z, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f);
        s[i] = a.softcap * fmaf(s[i], p, s[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) s[i] = a.softcap * tanhf(s[i]);
    }
  }
  if (slope != 0.f) {
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] -= slope * (float)dist(i);
  }
}

// One row and head over the keys [lo, hi] of its sequence, all of which it sees, by one warp on the CUDA cores: lane j scores every 32nd key, lane l owns the
// value columns l, l + 32, ...  For the rows whose sums were not finite, so it is never worth being fast.
template <int DV> struct PlainRow {
  float m, l, o[DV / 32];
};
template <int DK, int DV, int NQ>
__device__ __noinline__ PlainRow<DV> plain_row(const void* q, size_t q_at, const bf16* kc, size_t k_stride, const bf16* vc, size_t v_stride, int lo, int hi, int pos, float mul,
                                               float slope, float softcap) {
  const int lane = threadIdx.x & 31;
  PlainRow<DV> y;
  y.m = -INFINITY;
  y.l = 0.f;
#pragma unroll
  for (int c = 0; c < DV / 32; ++c) y.o[c] = 0.f;
  for (int j0 = lo; j0 <= hi; j0 += 32) {
    const int nk = min(32, hi + 1 - j0);
    float s = 0.f;
    if (lane < nk) {
      for (int d = 0; d < DK; ++d) {
        const float x = NQ == 1 ? __bfloat162float(reinterpret_cast<const bf16*>(q)[q_at + d]) : reinterpret_cast<const float*>(q)[q_at + d];
        s = fmaf(x, __bfloat162float(kc[(size_t)(j0 + lane) * k_stride + d]), s);
      }
      s *= mul;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      if (slope != 0.f) s -= slope * (float)(pos - j0 - lane);
    } else {
      s = -INFINITY;
    }
    const float m = fmaxf(y.m, warp_max(s)), base = m == -INFINITY ? 0.f : m, p = expf(s - base), al = expf(y.m - base);
    y.m = m;
    y.l = fmaf(y.l, al, warp_sum(p));
#pragma unroll
    for (int c = 0; c < DV / 32; ++c) y.o[c] *= al;
    for (int j = 0; j < nk; ++j) {
      const float w = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
      for (int c = 0; c < DV / 32; ++c) y.o[c] = fmaf(w, __bfloat162float(vc[(size_t)(j0 + j) * v_stride + lane + 32 * c]), y.o[c]);
    }
  }
  return y;
}

// The portion that holds the tile-th tile of ROWS rows, and the tile within it, among the portions of `least` to `most` rows (a whole warp asks); < 0: there are fewer tiles
template <int ROWS> __device__ __forceinline__ int portion_of(const int* __restrict__ segs, int nseg, int& tile, int least, int most) {
  const int lane = threadIdx.x & 31;
  int found = -1;
  for (int base = 0; base < nseg && found < 0; base += 32) {             // 32 portions at a time
    const int rows = base + lane < nseg ? segs[4 * (base + lane) + 3] : 0, n = rows >= least && rows <= most ? (rows + ROWS - 1) / ROWS : 0;
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, tile < upto);
    if (hit) {
      found = base + __ffs(hit) - 1;
      tile -= __shfl_sync(0xffffffffu, upto - n, __ffs(hit) - 1);
    } else {
      tile -= __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  return found;
}

}  // namespace
