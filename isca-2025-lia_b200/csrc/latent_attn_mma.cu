// Latent attention (latent_attn.cu) of portions of sequences on the tensor cores.  The rows of a portion share their keys, so the other
// order of the two projections is less work: Wuk and Wuv are applied once to the latents the portion sees (latent_expand_sm100.cu; latents of more than 512 or no whole 64 numbers: linear_mma.cu), and the rows attend to
// per-head keys and values -- 320 instead of 1088 multiply-adds per (row, key, head) at heads of 128 + 64 channels and latents of 512.  Nothing
// is held in fewer bits than in the latent space, where the carried queries, the weights and the weighted latents are fp32: the expanded keys
// and values are kept as three bf16 parts of their fp32 sums, and so are the rotated query parts and the softmax's weights (mma.cuh).  With bf16
// queries and bf16 rotated keys a score is three products of each part, a weighted value six (of the nine).
//
// Heads of 128 + 64 channels are latent_attn_sm100.cu's (2048 tokens, 16 heads on latents of 512: 4794 us in the latent space on the CUDA cores and 439 us for its two projections; 130 there with the
// expansion).  Here, for heads of 64 + 64, one block per (64 rows, head), warp by 16 rows, the scores becoming the weights' operand in registers; 32 keys per stage.  Keys and values are fetched in turn
// (the next keys while the values are taken in, the next values while the scores are made), so one stage is enough and several blocks share an SM.  Bound: tensor cores and shared-memory reads about
// equally.  With the expansion, latents of 512: 2048 tokens, 16 heads 252 us; 700 rows behind 300, 32 heads 141; 64 rows, 16 heads 14.
// Rows whose sums are not finite are formed again key by key at the end, as in window_attn_mma.cu: a masked key's weight of 0 still meets its value.
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include "latent_attn_rows.cuh"

int latent_expanded_tc(const ExpandedArgs& a, int tiles, long long latents, cudaStream_t stream);      // latent_attn_sm100.cu

// latent_expand_sm100.cu
bool latent_expand_takes(long long slot_stride, int D, int K, int N, int part);
int latent_expand(const bf16* cache, int D, const long long* first, const int* rows, int n, const bf16* W, bf16* C, long long ldc, int N, int K, int part, cudaStream_t stream);
// linear_mma.cu
int linear_mma_parts(const bf16* const* src, const int* rows, int n, long long lda, const bf16* W, bf16* C, long long ldc, int N, int K, int part, cudaStream_t stream);

namespace {

constexpr int BM = 64, BK = 32;

// 16-byte chunk c of row r in a tile of rows of CH (at least 8) chunks, turned by the row (window_attn_mma.cu)
template <int CH> __device__ __forceinline__ uint32_t at_chunk(uint32_t base, int r, int c) { return base + (uint32_t)(r * CH + (c ^ (r & 7))) * 16u; }

template <int DN, int DR> constexpr int expanded_smem() { return (BM * DN + 3 * BM * DR + 2 * 3 * BK * DN + BK * DR) * 2; }

template <int DN, int DR>
__global__ void __launch_bounds__(128, 2) latent_expanded_kernel(const __grid_constant__ ExpandedArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int QC = DN / 8, RC = DR / 8, NT = BK / 8;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t qn = smem_u32(smem), qr = qn + BM * DN * 2, kn = qr + 3 * BM * DR * 2, kr = kn + 3 * BK * DN * 2, vs = kr + BK * DR * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int h = a.h0 + blockIdx.x, tile = gridDim.y - 1 - blockIdx.y;            // a portion's longest histories start first
  int ip = 0;
  while (ip + 1 < a.np && tile >= a.p[ip + 1].tile0) ++ip;
  const Portion& pt = a.p[ip];
  const int skip = (tile - pt.tile0) * BM, row0 = pt.row0 + skip;
  const int rows = min(BM, pt.n - skip), pos0 = pt.pos0 + skip, pos_last = pos0 + rows - 1;
  const int jb = max(0, pos0 - a.window + 1);
  const size_t key_stride = (size_t)a.nh * 6 * DN;
  const bf16* keys = a.parts + (size_t)pt.part0 * key_stride + (size_t)blockIdx.x * 3 * DN;
  const bf16* vals = keys + (size_t)a.nh * 3 * DN;
  const bf16* key_rot = pt.kr;

  // three parts side by side in memory, three tiles in shared memory; keys behind the last are zero
  auto load_parts = [&](uint32_t dst, const bf16* src, int j0) {
    for (int e = threadIdx.x; e < BK * 3 * QC; e += 128) {
      const int j = e / (3 * QC), rest = e - j * 3 * QC, p = rest / QC, c = rest - p * QC;
      const bool in = j0 + j <= pos_last;
      cp_async16(at_chunk<QC>(dst + p * BK * DN * 2, j, c), src + (size_t)(in ? j0 + j : pos_last) * key_stride + rest * 8, in ? 16 : 0);
    }
  };
  auto load_keys = [&](int j0) {
    load_parts(kn, keys, j0);
    for (int e = threadIdx.x; e < BK * RC; e += 128) {
      const int j = e / RC, c = e - j * RC;
      const bool in = j0 + j <= pos_last;
      cp_async16(at_chunk<RC>(kr, j, c), key_rot + (size_t)(in ? j0 + j : pos_last) * a.kr_stride + c * 8, in ? 16 : 0);
    }
  };
  load_keys(jb);
  cp_async_commit();
  load_parts(vs, vals, jb);
  cp_async_commit();
  for (int e = threadIdx.x; e < BM * QC; e += 128) {
    const int r = e / QC, c = e - r * QC;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < rows) v = *reinterpret_cast<const uint4*>(a.q + (size_t)(row0 + r) * a.ldq + (size_t)h * (DN + DR) + c * 8);
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at_chunk<QC>(qn, r, c)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
  for (int e = threadIdx.x; e < BM * RC; e += 128) {
    const int r = e / RC, c = e - r * RC;
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f), w = u;
    if (r < rows) {
      const float4* src = reinterpret_cast<const float4*>(a.qr + ((size_t)(row0 + r) * a.H + h) * a.qr_stride + c * 8);
      u = src[0];
      w = src[1];
    }
    uint32_t p[3][4];
    split3(u.x, u.y, p[0][0], p[1][0], p[2][0]);
    split3(u.z, u.w, p[0][1], p[1][1], p[2][1]);
    split3(w.x, w.y, p[0][2], p[1][2], p[2][2]);
    split3(w.z, w.w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
    for (int s = 0; s < 3; ++s)
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at_chunk<RC>(qr + s * BM * DR * 2, r, c)), "r"(p[s][0]), "r"(p[s][1]), "r"(p[s][2]), "r"(p[s][3]) : "memory");
  }

  const int wpos = pos0 + warp * 16;
  const bool warp_on = warp * 16 < rows;
  float O[DN / 8][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < DN / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) O[n][i] = 0.f;

  const int ntile = (pos_last - jb) / BK + 1;
#pragma unroll 1
  for (int it = 0; it < ntile; ++it) {
    const int j0 = jb + it * BK;
    const bool on = warp_on && j0 <= wpos + 15 && j0 + BK - 1 >= wpos - a.window + 1;
    cp_async_wait<1>();
    __syncthreads();                                     // the keys (and, at first, the queries) are there
    // Two sums per score: the unrotated channels' high products, 16 channels at a time added in fp32, and all the rest -- its small parts first, then the
    // rotated channels' high products.  The tensor cores cut sums off below the 24th bit: with the high products of all channels in one chain the output of 16 to
    // 100 rows behind up to 1500 positions was off by 0.9 to 1.15 times what the latent space gives, now by 0.68 to 0.90 (2048 tokens: 490 -> 505 us; the chain for
    // portions of 256 rows and more alone, where it is exact enough: 490 us again, but portions of 401 to 250 rows in two launches 210 us instead of 154).
    float S[NT][4], S2[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) S[n][i] = S2[n][i] = 0.f;
    if (on) {
#pragma unroll
      for (int kk = 0; kk < DN / 16; ++kk) {
        uint32_t af[4];
        ldsm_x4(at_chunk<QC>(qn, warp * 16 + (lane & 15), 2 * kk + (lane >> 4)), af);
#pragma unroll
        for (int n = 0; n < NT; n += 2)
#pragma unroll
          for (int p = 2; p >= 0; --p) {
            uint32_t b[4];
            ldsm_x4(at_chunk<QC>(kn + p * BK * DN * 2, n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), b);
            if (p > 0) {
              mma_bf16(S2[n], af, b[0], b[1]);
              mma_bf16(S2[n + 1], af, b[2], b[3]);
            } else {
              float f[2][4];
              mma_bf16_first(f[0], af, b[0], b[1]);
              mma_bf16_first(f[1], af, b[2], b[3]);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                S[n][i] += f[0][i];
                S[n + 1][i] += f[1][i];
              }
            }
          }
      }
#pragma unroll
      for (int p0 = 1; p0 >= 0; --p0)
#pragma unroll
        for (int kk = 0; kk < DR / 16; ++kk) {
          uint32_t af[2][4];
#pragma unroll
          for (int p = p0; p <= 2 * p0; ++p) ldsm_x4(at_chunk<RC>(qr + p * BM * DR * 2, warp * 16 + (lane & 15), 2 * kk + (lane >> 4)), af[p - p0]);
#pragma unroll
          for (int n = 0; n < NT; n += 2) {
            uint32_t b[4];
            ldsm_x4(at_chunk<RC>(kr, n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), b);
#pragma unroll
            for (int p = 2 * p0; p >= p0; --p) {
              mma_bf16(S2[n], af[p - p0], b[0], b[1]);
              mma_bf16(S2[n + 1], af[p - p0], b[2], b[3]);
            }
          }
        }
    }
    __syncthreads();                                     // the keys may be overwritten
    if (it + 1 < ntile) load_keys(j0 + BK);
    cp_async_commit();
    float al[2] = {1.f, 1.f};
    uint32_t pw[BK / 16][3][4];
    if (on) {
      const bool whole = j0 + BK - 1 <= wpos && j0 >= wpos + 15 - a.window + 1;
      float mx[2] = {m_run[0], m_run[1]};
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int j = j0 + n * 8 + 2 * t + (i & 1), pos = wpos + g + (i >> 1) * 8;
          float sc = (S[n][i] + S2[n][i]) * a.scale;
          if (!whole && (j > pos || pos - j >= a.window)) sc = -INFINITY;
          S[n][i] = sc;
          mx[i >> 1] = fmaxf(mx[i >> 1], sc);
        }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], 1));
        mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], 2));
        const float base = mx[u] == -INFINITY ? 0.f : mx[u];
        al[u] = expf(m_run[u] - base);
        m_run[u] = mx[u];
        mx[u] = base;
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[n][i] = expf(S[n][i] - mx[i >> 1]);
        }
#pragma unroll
      for (int u = 0; u < 2; ++u) {                      // the stage's sum apart from the running one, like the values'
        float part = 0.f;
#pragma unroll
        for (int n = 0; n < NT; ++n) part += S[n][2 * u] + S[n][2 * u + 1];
        l_run[u] = fmaf(l_run[u], al[u], part);
      }
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
#pragma unroll
        for (int u = 0; u < 4; ++u) split3_finite(S[2 * kk + (u >> 1)][(u & 1) * 2], S[2 * kk + (u >> 1)][(u & 1) * 2 + 1], pw[kk][0][u], pw[kk][1][u], pw[kk][2][u]);
    }
    cp_async_wait<1>();
    __syncthreads();                                     // the values are there
    if (on) {
#pragma unroll
      for (int n = 0; n < DN / 8; n += 2) {
        float c[2][4], r[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[0][i] = c[1][i] = r[0][i] = r[1][i] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
#pragma unroll
          for (int v = 2; v >= 0; --v) {
            uint32_t b[4];
            ldsm_x4_trans(at_chunk<QC>(vs + v * BK * DN * 2, kk * 16 + (lane & 15), n + (lane >> 4)), b);
#pragma unroll
            for (int p = 2 - v; p >= 0; --p) {
              mma_bf16(p + v ? r[0] : c[0], pw[kk][p], b[0], b[1]);
              mma_bf16(p + v ? r[1] : c[1], pw[kk][p], b[2], b[3]);
            }
          }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) O[n + e][i] = fmaf(O[n + e][i], al[i >> 1], c[e][i] + r[e][i]);
      }
    }
    __syncthreads();                                     // the values may be overwritten
    if (it + 1 < ntile) load_parts(vs, vals, j0 + BK);
    cp_async_commit();
  }

  // gate over the softmax's denominator, the sink among its terms: everything relative to the larger of maximum and sink
  auto factor = [&](size_t row, float m, float l) {
    const float f = a.gate ? a.gate[row * a.H + h] : 1.0f;
    if (a.sink == nullptr) return f / l;
    const float top = fmaxf(m, a.sink[h]), e = expf(m - top);
    return f * (e / (l * e + expf(a.sink[h] - top)));
  };
  unsigned again[2];                                     // lanes whose row's sums are not finite
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    l_run[u] += __shfl_xor_sync(0xffffffffu, l_run[u], 1);
    l_run[u] += __shfl_xor_sync(0xffffffffu, l_run[u], 2);
    const int r = warp * 16 + g + u * 8;
    float probe = 0.f;                                   // NaN if a sum is not finite
#pragma unroll
    for (int n = 0; n < DN / 8; ++n) probe = fmaf(O[n][2 * u], 0.f, fmaf(O[n][2 * u + 1], 0.f, probe));
    again[u] = __ballot_sync(0xffffffffu, r < rows && probe != 0.f);
    if (r >= rows || ((again[u] >> (4 * g)) & 15u)) continue;
    const size_t row = row0 + r, at = (row * a.H + h) * DN;
    const float f = factor(row, m_run[u], l_run[u]);
#pragma unroll
    for (int n = 0; n < DN / 8; ++n) {
      const int ch = n * 8 + 2 * t;
      const float y0 = O[n][2 * u] * f, y1 = O[n][2 * u + 1] * f;
      if (a.out_f32) *reinterpret_cast<float2*>(reinterpret_cast<float*>(a.out) + at + ch) = make_float2(y0, y1);
      else *reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(a.out) + at + ch) = pack_bf16x2(y0, y1);
    }
  }
  if ((again[0] | again[1]) == 0u) return;
#pragma unroll 1
  for (int i = 0; i < 16; ++i) {
    if ((((i < 8 ? again[0] : again[1]) >> (4 * (i & 7))) & 15u) == 0u) continue;
    const size_t row = row0 + warp * 16 + i;
    const PlainRow<DN> y = plain_row<DN, DR>(a.q + row * a.ldq + (size_t)h * (DN + DR), a.qr + (row * a.H + h) * a.qr_stride, keys, vals, key_stride, key_rot, a.kr_stride,
                                             max(0, wpos + i - a.window + 1), wpos + i, a.scale);
    const float f = factor(row, y.m, y.l);
#pragma unroll
    for (int c = 0; c < DN / 32; ++c) {
      const size_t at = (row * a.H + h) * DN + lane + 32 * c;
      if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = y.o[c] * f;
      else reinterpret_cast<bf16*>(a.out)[at] = __float2bfloat16_rn(y.o[c] * f);
    }
  }
}

template <int DN, int DR> int run(const ExpandedArgs& a, int tiles, cudaStream_t stream) {
  constexpr int smem = expanded_smem<DN, DR>();
  LIA_CUDA(cudaFuncSetAttribute(latent_expanded_kernel<DN, DR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  lia_launch(latent_expanded_kernel<DN, DR>, dim3(a.nh, tiles), dim3(128), smem, stream, a);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

}  // namespace

// bytes of workspace for portions that see `latents` latents between them
extern "C" size_t lia_latent_expanded_workspace_bytes(long long latents, int H, int dim) { return (size_t)latents * H * 6 * dim * 2; }

extern "C" int lia_latent_attn_expanded(const void* q, int ldq, const float* qr, int qr_stride, const void* cache, long long slot_stride, const int* portions, int np,
                                        const void* w_ukv, const float* gate, const float* sink, void* out, int out_f32, void* workspace, int H, int dim,
                                        int rot, int kv_rank, int window, float scale, lia_stream_t stream_) {
  long long most = 0;                                              // what the caller's workspace holds: any 16 neighbouring portions
  for (int i = 0; portions && i < np; ++i) {
    long long sum = 0;
    for (int j = i; j < np && j < i + MAX_PORTIONS; ++j) {
      const int* p = portions + 4 * j;
      sum += p[1] + p[3] - (window > 0 && p[1] - window + 1 > 0 ? p[1] - window + 1 : 0);
    }
    if (sum > most) most = sum;
  }
  return lia_latent_attn_expanded_in(q, ldq, qr, qr_stride, cache, slot_stride, portions, np, w_ukv, gate, sink, out, out_f32, workspace,
                                     lia_latent_expanded_workspace_bytes(most, H, dim), H, dim, rot, kv_rank, window, scale, stream_);
}

// Portions go together while they are at most MAX_PORTIONS and their expanded keys and values fit the workspace; a portion that does not fit by itself goes in
// groups of heads.  Neither changes a bit of the result: every number is made by the same sums.
extern "C" int lia_latent_attn_expanded_in(const void* q, int ldq, const float* qr, int qr_stride, const void* cache, long long slot_stride, const int* portions, int np,
                                           const void* w_ukv, const float* gate, const float* sink, void* out, int out_f32, void* workspace, size_t workspace_bytes, int H,
                                           int dim, int rot, int kv_rank, int window, float scale, lia_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LIA_CHECK_ARG(q && qr && cache && portions && w_ukv && out && workspace && np > 0 && H > 0 && H <= 65535, "lia_latent_attn_expanded: bad arguments");
  LIA_CHECK_ARG((dim == 128 || dim == 64) && rot == 64 && kv_rank > 0 && kv_rank % 8 == 0, "lia_latent_attn_expanded: heads of %d + %d channels on latents of %d", dim, rot, kv_rank);
  const uintptr_t addr = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(qr) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(w_ukv) |
                         reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(workspace);
  LIA_CHECK_ARG(addr % 16 == 0 && ldq % 8 == 0 && ldq >= H * (dim + rot) && qr_stride % 4 == 0 && slot_stride % 8 == 0, "lia_latent_attn_expanded: addresses and rows must be whole 16 bytes");
  const int D = kv_rank + rot, tile_rows = dim == 128 ? 128 : BM;
  const size_t room = workspace_bytes / lia_latent_expanded_workspace_bytes(1, 1, dim);          // (latent, head) pairs
  if (window <= 0) window = 1 << 30;
  for (int first = 0; first < np;) {
    ExpandedArgs a{reinterpret_cast<const bf16*>(q), qr, reinterpret_cast<const bf16*>(workspace), gate, sink, out, D, ldq, qr_stride, H, 0, 0, window, out_f32, 0, scale, {}};
    const bf16* src[MAX_PORTIONS];
    long long at[MAX_PORTIONS];                                    // the same as rows of the cache
    int rows[MAX_PORTIONS], tiles = 0;
    long long latents = 0;
    while (first < np && a.np < MAX_PORTIONS) {
      const int* p = portions + 4 * first;                         // slot, first position, first row, rows
      LIA_CHECK_ARG(p[0] >= 0 && p[1] >= 0 && p[2] >= 0 && p[3] > 0, "lia_latent_attn_expanded: bad portion");
      const int base = p[1] - window + 1 > 0 ? p[1] - window + 1 : 0, seen = p[1] + p[3] - base, i = a.np;
      if (i > 0 && ((size_t)(latents + seen) * H > room || latents + seen > INT_MAX)) break;
      src[i] = reinterpret_cast<const bf16*>(cache) + (size_t)p[0] * slot_stride + (size_t)base * D;
      rows[i] = seen;
      at[i] = (long long)p[0] * (slot_stride / D) + base;
      a.p[i] = Portion{src[i] + kv_rank, p[2], p[3], p[1] - base, (int)latents, tiles};
      tiles += (p[3] + tile_rows - 1) / tile_rows;
      latents += seen;
      ++a.np;
      ++first;
    }
    LIA_CHECK_ARG(tiles <= 65535, "lia_latent_attn_expanded: too many rows");
    LIA_CHECK_ARG((size_t)latents <= room, "lia_latent_attn_expanded: a workspace of %zu bytes does not hold one head of %lld latents", workspace_bytes, latents);
    const int most = (size_t)latents * H <= room ? H : (int)(room / latents);
    const bf16* wk = reinterpret_cast<const bf16*>(w_ukv);
    bf16* ws = reinterpret_cast<bf16*>(workspace);
    for (a.h0 = 0; a.h0 < H; a.h0 += a.nh) {
      a.nh = most < H - a.h0 ? most : H - a.h0;
      const long long ldc = 6ll * a.nh * dim;
      const bool tc = latent_expand_takes(slot_stride, D, kv_rank, a.nh * dim, dim);
      auto expand = [&](const bf16* w, bf16* to, int N) {
        return tc ? latent_expand(reinterpret_cast<const bf16*>(cache), D, at, rows, a.np, w, to, ldc, N, kv_rank, dim, stream) : linear_mma_parts(src, rows, a.np, D, w, to, ldc, N, kv_rank, dim, stream);
      };
      int rc;
      if (a.nh == H) {
        rc = expand(wk, ws, 2 * H * dim);
      } else {
        rc = expand(wk + (size_t)a.h0 * dim * kv_rank, ws, a.nh * dim);
        if (rc == LIA_OK) rc = expand(wk + (size_t)(H + a.h0) * dim * kv_rank, ws + (size_t)3 * a.nh * dim, a.nh * dim);
      }
      if (rc == LIA_OK) rc = dim == 128 ? latent_expanded_tc(a, tiles, latents, stream) : run<64, 64>(a, tiles, stream);
      if (rc != LIA_OK) return rc;
    }
  }
  return LIA_OK;
}
