// Decode attention (one query token per sequence) over the time-major KV cache.
// Replaces attentions.py:395-399 (cat + permute + contiguous of the whole cache), 493-536
// (3 transposes, bmm, softmax, bmm) for tgt_len == 1.  No mask is applied (attentions.py:500).
//
// HBM-bound: every cached K and V element is read exactly once, in place, with 128-bit
// streaming loads (a (t,b,h) row is d*2 = 128/256 contiguous bytes); the reference moves
// ~5x those bytes.  Flash-decoding: grid = (B*H, splits); a CTA owns keys [t0,t1) of one
// (b,h).  Scores are staged in shared memory, softmax statistics use warp shuffles.
//
// Numerics mirror the reference when splits == 1 (the B=64 bench case):
//   s = bf16(q.k)  [bmm output], p = bf16(exp(s-max)/sum) [softmax(dtype=bf16)], ctx = bf16(sum_t p*v).
// With splits > 1 (small batches) the partial results are combined flash-decoding style
// in fp32 and p is not rounded per element (difference <= 1 bf16 ulp of p).
#include "common.cuh"

namespace {

constexpr int THREADS = 128;
constexpr int MAX_CHUNK = 4096;   // keys per CTA (scores kept in smem)

// UNROLL: rows in flight per lane.  Ten take 72 registers, seven CTAs an SM and 143 KB in flight there.  B=64 H=56 d=128 T=289:
// 77.8 us (6.8 TB/s); with 4, 6, 8, 12: 80.7, 77.8, 82.3, 84.6.  B=16 H=32 d=64 T=300, where few CTAs leave each its own
// latency to wait for: 9.7 us; with 4, 6, 8, 12: 15.4, 15.6, 13.8, 11.0.  B=96 H=32 d=128: 68 us; 79, 74, 70, 85.
// Four at a time with a wait for all of them before the next four, and nothing in flight during the softmax, took 90.9, 18.0
// and 89.9 us.  Which row a lane adds, and in which order, does not depend on this number.
template <int D, int UNROLL>
__global__ void __launch_bounds__(THREADS) attn_decode_kernel(const bf16* __restrict__ q, const bf16* __restrict__ kc,
                                                              const bf16* __restrict__ vc, bf16* __restrict__ out,
                                                              float* __restrict__ ws, int T, int H, int cache_batch,
                                                              int b0, int t_chunk, int splits) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int LPR = D / 8;        // lanes per cached row (each lane owns 8 dims = 16 bytes)
  constexpr int RPW = 32 / LPR;     // rows per warp iteration
  extern __shared__ float sc[];     // [t_chunk] scores -> probabilities
  __shared__ float red[4];
  __shared__ float accs[4][D];

  const int bh = blockIdx.x;
  const int b = bh / H;
  const int hh = bh - b * H;
  const int split = blockIdx.y;
  const int t0 = split * t_chunk;
  const int n = min(T, t0 + t_chunk) - t0;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int chunk = lane % LPR;
  const int rsub = lane / LPR;

  float qf[8];
  unpack8(__ldg(reinterpret_cast<const uint4*>(q + (size_t)bh * D + chunk * 8)), qf);
  const size_t row_stride = (size_t)cache_batch * H * D;
  const size_t base = ((size_t)(b0 + b) * H + hh) * D + chunk * 8 + (size_t)t0 * row_stride;

  // One list of rows, K's and then V's: a register is asked for again as soon as its row is used, so that UNROLL loads a lane
  // are on their way at all times, during the softmax between the passes too.
  constexpr int BATCH = 4 * RPW * UNROLL;
  uint4 row[UNROLL];
#pragma unroll
  for (int j = 0; j < UNROLL; ++j) {
    const int r = (j * 4 + warp) * RPW + rsub;
    if (r < n) row[j] = ldg_stream(kc + base + (size_t)r * row_stride);
  }

  // ---- phase A: s_t = bf16(q . k_t)
  for (int i = 0; i < n; i += BATCH) {
    const bool more = i + BATCH < n;
    const bf16* next = more ? kc + base : vc + base;
#pragma unroll
    for (int j = 0; j < UNROLL; ++j) {
      const int place = (j * 4 + warp) * RPW + rsub;
      const int r = i + place;
      float dot = 0.f;
      if (r < n) {
        float kf[8];
        unpack8(row[j], kf);
#pragma unroll
        for (int e = 0; e < 8; ++e) dot = fmaf(qf[e], kf[e], dot);
      }
      const int rn = more ? r + BATCH : place;
      if (rn < n) row[j] = ldg_stream(next + (size_t)rn * row_stride);
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (chunk == 0 && r < n) sc[r] = bf16r(dot);
    }
  }
  __syncthreads();

  // ---- softmax statistics over the chunk
  float m = -INFINITY;
  for (int i = threadIdx.x; i < n; i += THREADS) m = fmaxf(m, sc[i]);
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float l = 0.f;
  for (int i = threadIdx.x; i < n; i += THREADS) {
    const float e = expf(sc[i] - m);
    sc[i] = e;
    l += e;
  }
  l = warp_sum(l);
  if (lane == 0) red[warp] = l;
  __syncthreads();
  l = red[0] + red[1] + red[2] + red[3];
  if (splits == 1) {
    for (int i = threadIdx.x; i < n; i += THREADS) sc[i] = bf16r(sc[i] / l);
  }
  __syncthreads();

  // ---- phase B: ctx = sum_t p_t * v_t
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  for (int i = 0; i < n; i += BATCH) {
#pragma unroll
    for (int j = 0; j < UNROLL; ++j) {
      const int r = i + (j * 4 + warp) * RPW + rsub;
      if (r < n) {
        const float pj = sc[r];
        float vf[8];
        unpack8(row[j], vf);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(pj, vf[e], acc[e]);
      }
      if (r + BATCH < n) row[j] = ldg_stream(vc + base + (size_t)(r + BATCH) * row_stride);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
#pragma unroll
    for (int o = 16; o >= LPR; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  }
  if (rsub == 0) {
#pragma unroll
    for (int e = 0; e < 8; ++e) accs[warp][chunk * 8 + e] = acc[e];
  }
  __syncthreads();
  if (threadIdx.x < D) {
    const int e = threadIdx.x;
    const float o = accs[0][e] + accs[1][e] + accs[2][e] + accs[3][e];
    if (splits == 1) {
      out[(size_t)bh * D + e] = __float2bfloat16_rn(o);
    } else {
      float* dst = ws + ((size_t)bh * splits + split) * (D + 2);
      dst[2 + e] = o;
      if (e == 0) {
        dst[0] = m;
        dst[1] = l;
      }
    }
  }
}

// A short range's rows are all in flight from the start, and every lane goes through the places of those that are not there: the fewest of 2, 4 and 10 that hold the range.  With 2, 4, 10, and
// four at a time as above, us: B=96 H=56 d=128 T=8 9.6, 13.6, 23.7 (14.6), T=32 17.1, 16.3, 25.7 (19.5), T=48 23.1, 24.2, 27.9 (28.2); B=64 H=32 d=64 T=32 6.4, 7.0, 9.9 (8.2), T=64 9.7, 8.2, 11.3
// (11.3), T=80 12.2, 11.1, 11.9 (14.8).
template <int D> auto kernel_for(int range) {
  constexpr int STEP = 4 * 256 / D;          // rows of a CTA's lanes
  return range <= 2 * STEP ? attn_decode_kernel<D, 2> : range <= 4 * STEP ? attn_decode_kernel<D, 4> : attn_decode_kernel<D, 10>;
}

template <int D>
__global__ void attn_decode_combine_kernel(const float* __restrict__ ws, bf16* __restrict__ out, int splits) {
  pdl_launch_dependents();
  pdl_wait();
  const int bh = blockIdx.x;
  const int e = threadIdx.x;
  const float* src = ws + (size_t)bh * splits * (D + 2);
  float M = -INFINITY;
  for (int s = 0; s < splits; ++s) M = fmaxf(M, src[s * (D + 2)]);
  float L = 0.f, o = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float sc = expf(src[s * (D + 2)] - M);
    L += src[s * (D + 2) + 1] * sc;
    o += src[s * (D + 2) + 2 + e] * sc;
  }
  out[(size_t)bh * D + e] = __float2bfloat16_rn(o / L);
}

// CTAs per SM the split choice aims for.  Default 2: the unsharded shapes (B * H in the thousands) keep one CTA per (b, h)
// and with it the reference's per-element rounding of p.  A caller whose rank keeps only H / world heads asks for more
// (`splits` = -6 from the tensor-parallel model): at B * H = 448 (OPT-30B, TP8) one CTA per (b, h) left 3 latency-bound CTAs
// per SM -- 24 us for 9.5 us of K/V bytes -- and two key ranges per (b, h) took a 16-layer stack at TP8 shapes from 152.5 to
// 140.0 us per layer (profiles/README.md).  LIA_ATTN_CTAS_PER_SM overrides the default of the automatic choice (A/B runs).
int pick_splits(int B, int H, int T, int per_sm) {
  int splits = (T + MAX_CHUNK - 1) / MAX_CHUNK;
  if (per_sm <= 0) {
    static int dflt = 0;
    if (dflt == 0) {
      const char* e = getenv("LIA_ATTN_CTAS_PER_SM");
      dflt = (e && atoi(e) > 0) ? atoi(e) : 2;
    }
    per_sm = dflt;
  }
  const int want = (per_sm * lia_sm_count() + B * H - 1) / (B * H);
  const int cap = T / 128 > 1 ? T / 128 : 1;                     // keep >= 128 keys per CTA
  int s = want < cap ? want : cap;
  if (s > 32) s = 32;
  return s > splits ? s : splits;
}

}  // namespace

extern "C" size_t lia_attn_decode_workspace_bytes(int B, int H, int d, int max_splits) {
  if (B <= 0 || H <= 0 || d <= 0) return 0;
  if (max_splits <= 0) max_splits = 32;
  return (size_t)B * H * max_splits * (d + 2) * sizeof(float);
}

extern "C" int lia_attn_decode_bf16(const void* q, const void* k_cache, const void* v_cache, void* out, int B, int H,
                                    int T, int d, int cache_batch, int b0, int splits, void* workspace,
                                    size_t workspace_bytes, lia_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LIA_CHECK_ARG(q && k_cache && v_cache && out, "lia_attn_decode_bf16: null pointer");
  LIA_CHECK_ARG(d == 64 || d == 128, "lia_attn_decode_bf16: head_dim must be 64 or 128 (got %d)", d);
  LIA_CHECK_ARG(B > 0 && H > 0 && T > 0, "lia_attn_decode_bf16: B,H,T must be positive");
  LIA_CHECK_ARG(b0 >= 0 && b0 + B <= cache_batch, "lia_attn_decode_bf16: batch window [%d,%d) outside cache batch %d", b0, b0 + B, cache_batch);
  if (splits <= 0) splits = pick_splits(B, H, T, -splits);   // 0: automatic; -n: automatic, aiming for n CTAs per SM
  if (splits > 1 && (workspace == nullptr || workspace_bytes < (size_t)B * H * splits * (d + 2) * sizeof(float))) {
    splits = (T + MAX_CHUNK - 1) / MAX_CHUNK;   // fall back to the fewest splits that fit shared memory
    LIA_CHECK_ARG(splits == 1, "lia_attn_decode_bf16: T=%d needs a workspace of lia_attn_decode_workspace_bytes()", T);
  }
  int t_chunk = (T + splits - 1) / splits;
  splits = (T + t_chunk - 1) / t_chunk;        // no empty splits
  LIA_CHECK_ARG(t_chunk <= MAX_CHUNK, "lia_attn_decode_bf16: chunk too large");
  const dim3 grid(B * H, splits);
  const size_t smem = (size_t)t_chunk * sizeof(float);
  const bf16* qp = reinterpret_cast<const bf16*>(q);
  const bf16* kp = reinterpret_cast<const bf16*>(k_cache);
  const bf16* vp = reinterpret_cast<const bf16*>(v_cache);
  bf16* op = reinterpret_cast<bf16*>(out);
  float* wsp = reinterpret_cast<float*>(workspace);
  if (d == 128) {
    lia_launch(kernel_for<128>(t_chunk), dim3(grid), dim3(THREADS), smem, stream, qp, kp, vp, op, wsp, T, H, cache_batch, b0, t_chunk, splits);
    LIA_LAUNCH_CHECK();
    if (splits > 1) lia_launch(attn_decode_combine_kernel<128>, dim3(B * H), dim3(128), 0, stream, wsp, op, splits);
  } else {
    lia_launch(kernel_for<64>(t_chunk), dim3(grid), dim3(THREADS), smem, stream, qp, kp, vp, op, wsp, T, H, cache_batch, b0, t_chunk, splits);
    LIA_LAUNCH_CHECK();
    if (splits > 1) lia_launch(attn_decode_combine_kernel<64>, dim3(B * H), dim3(64), 0, stream, wsp, op, splits);
  }
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}
