// Softmax attention over cached keys and values (window_attn.cu) on the tensor cores, for bf16 caches with heads of 64, 128 or 256
// channels.  Nothing is held in fewer bits than on the CUDA cores: the caches are bf16 as they are, fp32 queries and the softmax's
// weights enter as three bf16 parts (mma.cuh), scores and sums are fp32.
//
//   prompt:  one block per (64 rows of one portion, query head); with heads of 128 + 128 channels only for many short portions (lia_window_prompt_form), the others are
//            window_attn_sm100.cu's.  Bound: tensor cores and the softmax's instructions about equally -- mma.sync m16n8k16, one product for
//            q . k (three for fp32 queries) and three for the weights times the values.  A warp owns 16 rows: its 16 x 32 scores become the
//            weights' operand in registers, so nothing but keys and values passes through shared memory; those come by cp.async, two stages of 32 keys (64 keys need 255 registers: two blocks per SM instead of three, 185 instead of 159 us).
//            2048 tokens, 16 heads of 128 on 8 key heads, window 1024, soft cap: 1183 -> 136 us; the whole history, fp32 queries: 1713 -> 182 us (66 and 63 us there).
//   decode:  one block per (row, up to 8 query heads of one key/value head, range of keys).  Bound: HBM.  The heads of a group are the rows of
//            the matrix instruction and a warp reads every cached row once for all of them, straight from global memory into operand
//            registers: channels and value columns may be taken in any order as long as q and the output follow it, so a lane's 16
//            bytes of a key row are two operands and those of two value rows interleave into eight.  No shared memory until the
//            warps of a block (every fourth 16 keys each) meet at the end.  16 sequences of 1902 positions, 16 heads on 8 key heads: 163 ->
//            34 us (3.7 TB/s).
// The tensor cores cut sums off below the 24th bit instead of rounding them.  Sums over one stage are therefore made apart and added to the
// running ones in fp32: the error against 64 bits is 0.4 to 0.8 times that of the FMA chains (one running sum over 1700 keys: 5 times).
// Numbers that are not finite do not survive this: a masked key of the stage has weight 0 and still meets its value, and a part of a split weight is 0 or has
// the other sign.  Sums that are not finite stay so to the end, so it is there that such rows are found and formed again key by key (plain_row).
#include <limits.h>

#include "window_attn_rows.cuh"

int window_prompt_tc(const void* q, int ldq, const bf16* kcache, long long kss, const bf16* vcache, long long vss, const int* meta, const int* segs, int nseg, const WindowExtras& x, bf16* out,
                     int M, const WindowArgs& a, int least, int tiles, cudaStream_t stream);      // window_attn_sm100.cu

namespace {

constexpr int BM = 64;                 // rows of a prompt block

// 16-byte chunk c of row r in a tile of rows of CH chunks: the chunk's place is turned by the row, so that ldmatrix (8 rows, one chunk)
// touches all banks
template <int CH> __device__ __forceinline__ uint32_t at_chunk(uint32_t base, int r, int c) { return base + (uint32_t)(r * CH + (c ^ (r & 7))) * 16u; }

// rows j0 .. j0 + BK - 1 of a cache (head offset and row stride in elements); rows behind `last` are zero
template <int D, int BK> __device__ __forceinline__ void load_tile(uint32_t dst, const bf16* rows, size_t stride, int j0, int last) {
  constexpr int CH = D / 8;
  for (int e = threadIdx.x; e < BK * CH; e += 128) {
    const int j = e / CH, c = e - j * CH;
    const bool in = j0 + j <= last;
    cp_async16(at_chunk<CH>(dst, j, c), rows + (size_t)(in ? j0 + j : last) * stride + c * 8, in ? 16 : 0);
  }
}

template <int DK, int DV, int NQ> struct PromptShape {
  static constexpr int BK = 32;
  static constexpr int SMEM = NQ * BM * DK * 2 + 2 * BK * (DK + DV) * 2;
};

// NQ = 1: bf16 queries; 3: fp32 queries in three parts.  segs[s] = {slot, first position, first row, rows}; null: one portion that meta's first
// row begins (tiles whose rows do not continue it are taken row by row).  Portions of more than `most` rows are another kernel's.  blockIdx.y counts the portions' tiles from the last to the
// first: the longest histories start first.
template <int DK, int DV, int NQ>
__global__ void __launch_bounds__(128, (DV <= 128 && NQ == 1) ? 3 : 2) window_prompt_kernel(const void* __restrict__ q, int ldq, const bf16* __restrict__ kcache, long long k_slot_stride,
                                                            const bf16* __restrict__ vcache, long long v_slot_stride, const int* __restrict__ meta,
                                                            const int* __restrict__ segs, int nseg, int most, WindowExtras x, bf16* __restrict__ out, int M, WindowArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int BK = PromptShape<DK, DV, NQ>::BK, QC = DK / 8, VC = DV / 8, NT = BK / 8;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t qs = smem_u32(smem), ks = qs + NQ * BM * DK * 2, vs = ks + 2 * BK * DK * 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int tile = gridDim.y - 1 - blockIdx.y, slot, pos0, row0, rows;
  if (segs == nullptr) {
    slot = meta[0]; pos0 = meta[1]; row0 = 0; rows = M;
    if (tile * BM >= rows) return;
  } else {
    const int found = portion_of<BM>(segs, nseg, tile, 1, most);
    if (found < 0) return;
    slot = segs[4 * found]; pos0 = segs[4 * found + 1]; row0 = segs[4 * found + 2]; rows = segs[4 * found + 3];
  }
  const int h = blockIdx.x, kg = h / (a.H / a.G), vg = kg / a.v_div, Gv = a.G / a.v_div;
  row0 += tile * BM;
  pos0 += tile * BM;
  rows = min(BM, rows - tile * BM);
  const size_t k_stride = (size_t)a.G * DK, v_stride = (size_t)Gv * DV;
  const float mul = a.scale * (x.temp ? x.temp[h] : 1.0f), slope = x.slopes ? x.slopes[h] : 0.f;
  auto by_itself = [&](size_t row, int slot_, int pos) {               // one row by one warp
    const PlainRow<DV> y = plain_row<DK, DV, NQ>(q, row * ldq + (size_t)h * DK, kcache + (size_t)slot_ * k_slot_stride + (size_t)kg * DK, k_stride,
                                                 vcache + (size_t)slot_ * v_slot_stride + (size_t)vg * DV, v_stride, first_key(a, pos), pos, pos, mul, slope, a.softcap);
    const float invl = 1.0f / (y.l + (x.sink ? expf(x.sink[h] - y.m) : 0.f));
#pragma unroll
    for (int c = 0; c < DV / 32; ++c) {
      const int ch = lane + 32 * c;
      store_out(out, (row * a.H + h) * DV + ch, y.o[c] * invl * gate_of<bf16>(x, a, row, h, ch), a);
    }
  };
  if (segs == nullptr) {                                 // what meta says counts: rows that do not continue one sequence go one by one
    bool run = true;
    if ((int)threadIdx.x < rows) run = meta[2 * (row0 + threadIdx.x)] == slot && meta[2 * (row0 + threadIdx.x) + 1] == pos0 + (int)threadIdx.x;
    if (!__syncthreads_and(run)) {
#pragma unroll 1
      for (int r = warp; r < rows; r += 4) by_itself(row0 + r, meta[2 * (row0 + r)], meta[2 * (row0 + r) + 1]);
      return;
    }
  }
  const int pos_last = pos0 + rows - 1, jb = first_key(a, pos0);
  const bf16* kc = kcache + (size_t)slot * k_slot_stride + (size_t)kg * DK;
  const bf16* vc = vcache + (size_t)slot * v_slot_stride + (size_t)vg * DV;
  load_tile<DK, BK>(ks, kc, k_stride, jb, pos_last);
  load_tile<DV, BK>(vs, vc, v_stride, jb, pos_last);
  cp_async_commit();
  for (int e = threadIdx.x; e < BM * QC; e += 128) {
    const int r = e / QC, c = e - r * QC;
    uint32_t part[3][4];
#pragma unroll
    for (int s = 0; s < 3; ++s)
#pragma unroll
      for (int i = 0; i < 4; ++i) part[s][i] = 0u;
    if (r < rows) {
      const size_t at = (size_t)(row0 + r) * ldq + (size_t)h * DK + c * 8;
      if constexpr (NQ == 1) {
        const uint4 v = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(q) + at);
        part[0][0] = v.x; part[0][1] = v.y; part[0][2] = v.z; part[0][3] = v.w;
      } else {
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q) + at);
        const float4 u = src[0], w = src[1];
        split3(u.x, u.y, part[0][0], part[1][0], part[2][0]);
        split3(u.z, u.w, part[0][1], part[1][1], part[2][1]);
        split3(w.x, w.y, part[0][2], part[1][2], part[2][2]);
        split3(w.z, w.w, part[0][3], part[1][3], part[2][3]);
      }
    }
#pragma unroll
    for (int s = 0; s < NQ; ++s)
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at_chunk<QC>(qs + s * BM * DK * 2, r, c)), "r"(part[s][0]), "r"(part[s][1]),
                   "r"(part[s][2]), "r"(part[s][3]) : "memory");
  }

  const int wpos = pos0 + warp * 16;                     // position of the warp's first row
  const bool warp_on = warp * 16 < rows;
  float O[DV / 8][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < DV / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) O[n][i] = 0.f;

  const int ntile = (pos_last - jb) / BK + 1;
  for (int it = 0; it < ntile; ++it) {
    const int j0 = jb + it * BK;
    const uint32_t kt = ks + (it & 1) * BK * DK * 2, vt = vs + (it & 1) * BK * DV * 2;
    if (it + 1 < ntile) {
      load_tile<DK, BK>(ks + ((it + 1) & 1) * BK * DK * 2, kc, k_stride, j0 + BK, pos_last);
      load_tile<DV, BK>(vs + ((it + 1) & 1) * BK * DV * 2, vc, v_stride, j0 + BK, pos_last);
    }
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (warp_on && j0 <= wpos + 15 && j0 + BK - 1 >= first_key(a, wpos)) {
      // two sums per score, added at the end: the tensor cores cut their sums off below the 24th bit, so chains are kept short and the
      // small parts of fp32 queries, whose cut-off bits lie far below, have their own
      float S[NT][4], S2[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[n][i] = S2[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < DK / 16; ++kk) {
        uint32_t af[NQ][4];
#pragma unroll
        for (int s = 0; s < NQ; ++s) ldsm_x4(at_chunk<QC>(qs + s * BM * DK * 2, warp * 16 + (lane & 15), 2 * kk + (lane >> 4)), af[s]);
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
          uint32_t b[4];
          ldsm_x4(at_chunk<QC>(kt, n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), b);
          if constexpr (NQ == 1) {
            mma_bf16(kk & 1 ? S2[n] : S[n], af[0], b[0], b[1]);
            mma_bf16(kk & 1 ? S2[n + 1] : S[n + 1], af[0], b[2], b[3]);
          } else {
#pragma unroll
            for (int s = 2; s >= 0; --s) {
              mma_bf16(s ? S2[n] : S[n], af[s], b[0], b[1]);
              mma_bf16(s ? S2[n + 1] : S[n + 1], af[s], b[2], b[3]);
            }
          }
        }
      }
      const bool whole = j0 + BK - 1 <= wpos && j0 >= first_key(a, wpos + 15);      // every row of the warp sees every key of the stage
      const int lo0 = first_key(a, wpos + g), lo1 = first_key(a, wpos + g + 8);
      float sc[NT * 4];
#pragma unroll
      for (int e = 0; e < NT * 4; ++e) sc[e] = S[e >> 2][e & 3] + S2[e >> 2][e & 3];
      const int ahead = wpos + g - j0 - 2 * t;                                       // position of the thread's first row less its first key's
      finish_scores(sc, mul, a, slope, [&](int e) { return ahead + ((e >> 1) & 1) * 8 - (e >> 2) * 8 - (e & 1); });
      float mx[2] = {m_run[0], m_run[1]};
#pragma unroll
      for (int e = 0; e < NT * 4; ++e) {
        const int u = (e >> 1) & 1, j = j0 + (e >> 2) * 8 + 2 * t + (e & 1);
        if (!whole && (j > wpos + g + u * 8 || j < (u ? lo1 : lo0))) sc[e] = -INFINITY;
        mx[u] = fmaxf(mx[u], sc[e]);
      }
      float al[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], 1));
        mx[u] = fmaxf(mx[u], __shfl_xor_sync(0xffffffffu, mx[u], 2));
        const float base = mx[u] == -INFINITY ? 0.f : mx[u];                       // no key seen so far
        al[u] = expf(m_run[u] - base);
        m_run[u] = mx[u];
        mx[u] = base;
        l_run[u] *= al[u];
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[n][i] = expf(sc[4 * n + i] - mx[i >> 1]);
          l_run[i >> 1] += S[n][i];
        }
      uint32_t p[BK / 16][3][4];
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
#pragma unroll
        for (int u = 0; u < 4; ++u) split3_finite(S[2 * kk + (u >> 1)][(u & 1) * 2], S[2 * kk + (u >> 1)][(u & 1) * 2 + 1], p[kk][0][u], p[kk][1][u], p[kk][2][u]);
#pragma unroll
      for (int n = 0; n < DV / 8; n += 2) {              // a stage's sums apart from the running ones (short chains again)
        float c[2][4], r[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[0][i] = c[1][i] = r[0][i] = r[1][i] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk) {
          uint32_t b[4];
          ldsm_x4_trans(at_chunk<VC>(vt, kk * 16 + (lane & 15), n + (lane >> 4)), b);
#pragma unroll
          for (int s = 2; s >= 0; --s) {
            mma_bf16(s ? r[0] : c[0], p[kk][s], b[0], b[1]);
            mma_bf16(s ? r[1] : c[1], p[kk][s], b[2], b[3]);
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) O[n + e][i] = fmaf(O[n + e][i], al[i >> 1], c[e][i] + r[e][i]);
      }
    }
    __syncthreads();                                     // the stage may be overwritten
  }

  unsigned again[2];                                     // lanes whose row's sums are not finite
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    l_run[u] += __shfl_xor_sync(0xffffffffu, l_run[u], 1);
    l_run[u] += __shfl_xor_sync(0xffffffffu, l_run[u], 2);
    const int r = warp * 16 + g + u * 8;
    float probe = 0.f;                                   // NaN if a sum is not finite
#pragma unroll
    for (int n = 0; n < DV / 8; ++n) probe = fmaf(O[n][2 * u], 0.f, fmaf(O[n][2 * u + 1], 0.f, probe));
    again[u] = __ballot_sync(0xffffffffu, r < rows && probe != 0.f);
    if (r >= rows || ((again[u] >> (4 * g)) & 15u)) continue;
    const float invl = 1.0f / (l_run[u] + (x.sink ? expf(x.sink[h] - m_run[u]) : 0.f));
    const size_t row = row0 + r, at = (row * a.H + h) * DV;
#pragma unroll
    for (int n = 0; n < DV / 8; ++n) {
      const int ch = n * 8 + 2 * t;
      const float y0 = O[n][2 * u] * invl * gate_of<bf16>(x, a, row, h, ch), y1 = O[n][2 * u + 1] * invl * gate_of<bf16>(x, a, row, h, ch + 1);
      if (a.out_f32) *reinterpret_cast<float2*>(reinterpret_cast<float*>(out) + at + ch) = make_float2(y0, y1);
      else *reinterpret_cast<uint32_t*>(out + at + ch) = pack_bf16x2(y0, y1);
    }
  }  if ((again[0] | again[1]) == 0u) return;
#pragma unroll 1
  for (int i = 0; i < 16; ++i) {
    if ((((i < 8 ? again[0] : again[1]) >> (4 * (i & 7))) & 15u) == 0u) continue;
    by_itself(row0 + warp * 16 + i, slot, wpos + i);
  }
}

// One row, HB (at most 8) query heads of one key/value head, the blockIdx.y-th of nsplit ranges of its keys; the block's four warps take 16 keys
// at a time in turn.  nsplit > 1: unnormalised sums and (max, sum) to part / part_ml, as in window_attn.cu.
template <int DK, int DV, int NQ>
__global__ void __launch_bounds__(128) window_decode_kernel(const void* __restrict__ q, int ldq, const bf16* __restrict__ kcache, long long k_slot_stride,
                                                            const bf16* __restrict__ vcache, long long v_slot_stride, const int* __restrict__ meta,
                                                            WindowExtras x, bf16* __restrict__ out, float* __restrict__ part, float2* __restrict__ part_ml,
                                                            WindowArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int KC = DK / 32, VU = DV / 64;              // 16-byte chunks of a key row / value row per lane
  extern __shared__ __align__(16) float sums[];          // [4 warps][8 heads][DV]
  __shared__ float2 ml[4][8];
  const int nhb = a.H / a.HB, row = blockIdx.x / nhb, h0 = (blockIdx.x - row * nhb) * a.HB, z = blockIdx.y;
  const int kg = h0 / (a.H / a.G), vg = kg / a.v_div, Gv = a.G / a.v_div;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int slot = meta[2 * row], pos = meta[2 * row + 1], lo = first_key(a, pos);
  const bf16* kc = kcache + (size_t)slot * k_slot_stride + (size_t)kg * DK;
  const bf16* vc = vcache + (size_t)slot * v_slot_stride + (size_t)vg * DV;
  const size_t k_stride = (size_t)a.G * DK, v_stride = (size_t)Gv * DV;

  // Operand of the queries: lane (g, t) holds head g at channels 8 c .. 8 c + 7, c = 4 s + t, two k-steps per chunk.  The instruction has 16
  // rows for 8 heads, so rows 8 .. 15 carry the middle part of what rows 0 .. 7 carry the high part of: one product for both.
  uint32_t qf[NQ][KC][4];
#pragma unroll
  for (int s = 0; s < KC; ++s) {
#pragma unroll
    for (int n = 0; n < NQ; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) qf[n][s][i] = 0u;
    if (g < a.HB) {
      const size_t at = (size_t)row * ldq + (size_t)(h0 + g) * DK + (s * 4 + t) * 8;
      if constexpr (NQ == 1) {
        const uint4 v = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(q) + at);
        qf[0][s][0] = v.x; qf[0][s][1] = v.y; qf[0][s][2] = v.z; qf[0][s][3] = v.w;
      } else {
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q) + at);
        const float4 u = src[0], w = src[1];
        split3(u.x, u.y, qf[0][s][0], qf[1][s][0], qf[2][s][0]);
        split3(u.z, u.w, qf[0][s][1], qf[1][s][1], qf[2][s][1]);
        split3(w.x, w.y, qf[0][s][2], qf[1][s][2], qf[2][s][2]);
        split3(w.z, w.w, qf[0][s][3], qf[1][s][3], qf[2][s][3]);
      }
    }
  }
  const int h = h0 + min(g, a.HB - 1);
  const float mul = a.scale * (x.temp ? x.temp[h] : 1.0f), slope = x.slopes ? x.slopes[h] : 0.f;
  float O[VU * 8][2], m_run = -INFINITY, l_run = 0.f;
#pragma unroll
  for (int n = 0; n < VU * 8; ++n) O[n][0] = O[n][1] = 0.f;

  const int tiles = (pos - lo) / 16 + 1, per = (tiles + a.nsplit - 1) / a.nsplit, t_end = min(tiles, (z + 1) * per);
  // keys g, g + 8; values of keys 2t, 2t + 1, 2t + 8, 2t + 9 (a key behind the last: the last).  The next keys are on their way while this
  // tile's values are taken in.
  uint4 kv[2][KC];
  auto load_keys = [&](int it) {
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int s = 0; s < KC; ++s) kv[u][s] = ldg_stream(kc + (size_t)min(lo + it * 16 + g + 8 * u, pos) * k_stride + (s * 4 + t) * 8);
  };
  if (z * per + warp < t_end) load_keys(z * per + warp);
#pragma unroll 1
  for (int it = z * per + warp; it < t_end; it += 4) {
    const int j0 = lo + it * 16;
    constexpr int VH = VU < 2 ? VU : 2;                  // value chunks in flight: 128 columns
    uint4 vv[4][VH];
    auto load_values = [&](int first) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int s = 0; s < VH; ++s)
          vv[u][s] = ldg_stream(vc + (size_t)min(j0 + 2 * t + (u & 1) + (u >> 1) * 8, pos) * v_stride + (g + 8 * (first + s)) * 8);
    };
    load_values(0);
    float S[2][2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float c[4] = {0.f, 0.f, 0.f, 0.f}, r[4] = {0.f, 0.f, 0.f, 0.f};        // as in the prompt kernel: short sums
#pragma unroll
      for (int s = 0; s < KC; ++s) {
        if constexpr (NQ == 1) {
          const uint32_t a0[4] = {qf[0][s][0], 0u, qf[0][s][1], 0u}, a1[4] = {qf[0][s][2], 0u, qf[0][s][3], 0u};
          mma_bf16(s & 1 ? r : c, a0, kv[u][s].x, kv[u][s].y);
          mma_bf16(s & 1 ? r : c, a1, kv[u][s].z, kv[u][s].w);
        } else {
          const uint32_t a0[4] = {qf[0][s][0], qf[1][s][0], qf[0][s][1], qf[1][s][1]}, a1[4] = {qf[0][s][2], qf[1][s][2], qf[0][s][3], qf[1][s][3]};
          const uint32_t l0[4] = {qf[2][s][0], 0u, qf[2][s][1], 0u}, l1[4] = {qf[2][s][2], 0u, qf[2][s][3], 0u};
          mma_bf16(r, l0, kv[u][s].x, kv[u][s].y);
          mma_bf16(r, l1, kv[u][s].z, kv[u][s].w);
          mma_bf16(c, a0, kv[u][s].x, kv[u][s].y);
          mma_bf16(c, a1, kv[u][s].z, kv[u][s].w);
        }
      }
      S[u][0] = c[0] + (c[2] + r[0]);
      S[u][1] = c[1] + (c[3] + r[1]);
    }
    if (it + 4 < t_end) load_keys(it + 4);
    float sc[4] = {S[0][0], S[0][1], S[1][0], S[1][1]}, mx = m_run;
    const int ahead = pos - j0 - 2 * t;
    finish_scores(sc, mul, a, slope, [&](int e) { return ahead - (e >> 1) * 8 - (e & 1); });
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (j0 + (e >> 1) * 8 + 2 * t + (e & 1) > pos) sc[e] = -INFINITY;
      mx = fmaxf(mx, sc[e]);
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float base = mx == -INFINITY ? 0.f : mx, al = expf(m_run - base);
    m_run = mx;
    l_run *= al;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        S[u][i] = expf(sc[2 * u + i] - base);
        l_run += S[u][i];
      }
    uint32_t ph[4], pl[4] = {0u, 0u, 0u, 0u};            // high part above the middle part; low part
#pragma unroll
    for (int u = 0; u < 2; ++u) split3_finite(S[u][0], S[u][1], ph[2 * u], ph[2 * u + 1], pl[2 * u]);
#pragma unroll
    for (int first = 0; first < VU; first += VH) {
      if (first > 0) load_values(first);
#pragma unroll
      for (int s = 0; s < VH; ++s)
#pragma unroll
        for (int w = 0; w < 4; ++w) {                    // value columns 8 (g + 8 s) + 2 w and + 2 w + 1
          const uint32_t r0 = (&vv[0][s].x)[w], r1 = (&vv[1][s].x)[w], r2 = (&vv[2][s].x)[w], r3 = (&vv[3][s].x)[w];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t sel = e ? 0x7632u : 0x5410u, b0 = __byte_perm(r0, r1, sel), b1 = __byte_perm(r2, r3, sel);
            float* o = O[(first + s) * 8 + 2 * w + e];
            float c[4] = {0.f, 0.f, 0.f, 0.f}, r[4] = {0.f, 0.f, 0.f, 0.f};
            mma_bf16(r, pl, b0, b1);
            mma_bf16(c, ph, b0, b1);
            o[0] = fmaf(o[0], al, c[0] + (c[2] + r[0]));
            o[1] = fmaf(o[1], al, c[1] + (c[3] + r[1]));
          }
        }
    }
  }

  l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
  l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
  if (t == 0) ml[warp][g] = make_float2(m_run, l_run);
#pragma unroll
  for (int s = 0; s < VU; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i) {                        // columns 8 (2 t + i + 8 s) + e
      float4* dst = reinterpret_cast<float4*>(sums + (warp * 8 + g) * DV + 8 * (2 * t + i + 8 * s));
      dst[0] = make_float4(O[s * 8][i], O[s * 8 + 1][i], O[s * 8 + 2][i], O[s * 8 + 3][i]);
      dst[1] = make_float4(O[s * 8 + 4][i], O[s * 8 + 5][i], O[s * 8 + 6][i], O[s * 8 + 7][i]);
    }
  float probe = 0.f;                                     // NaN if a sum is not finite
#pragma unroll
  for (int n = 0; n < VU * 8; ++n) probe = fmaf(O[n][0], 0.f, fmaf(O[n][1], 0.f, probe));
  if (__syncthreads_or(probe != 0.f)) {                  // the whole range again, a head per warp
#pragma unroll 1
    for (int hh = warp; hh < a.HB; hh += 4) {
      const int hq = h0 + hh;
      const PlainRow<DV> y = plain_row<DK, DV, NQ>(q, (size_t)row * ldq + (size_t)hq * DK, kc, k_stride, vc, v_stride, lo + z * per * 16, min(pos, lo + t_end * 16 - 1), pos,
                                                   a.scale * (x.temp ? x.temp[hq] : 1.0f), x.slopes ? x.slopes[hq] : 0.f, a.softcap);
      const size_t rh = (size_t)row * a.H + hq;
      const float invl = 1.0f / (y.l + (x.sink ? expf(x.sink[hq] - y.m) : 0.f));
#pragma unroll
      for (int c = 0; c < DV / 32; ++c) {
        const int ch = lane + 32 * c;
        if (a.nsplit == 1) store_out(out, rh * DV + ch, y.o[c] * invl * gate_of<bf16>(x, a, row, hq, ch), a);
        else part[(rh * a.nsplit + z) * DV + ch] = y.o[c];
      }
      if (a.nsplit > 1 && lane == 0) part_ml[rh * a.nsplit + z] = make_float2(y.m, y.l);
    }
    return;
  }
  for (int e = threadIdx.x; e < a.HB * DV; e += 128) {
    const int hh = e / DV, ch = e - hh * DV;
    float m = -INFINITY, l = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) m = fmaxf(m, ml[w][hh].x);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      if (ml[w][hh].y != 0.f) {                          // 0: the warp saw no key; a NaN is kept
        const float f = expf(ml[w][hh].x - m);
        l = fmaf(ml[w][hh].y, f, l);
        o = fmaf(sums[(w * 8 + hh) * DV + ch], f, o);
      }
    }
    const size_t rh = (size_t)row * a.H + h0 + hh;
    if (a.nsplit == 1) {
      const float invl = 1.0f / (l + (x.sink ? expf(x.sink[h0 + hh] - m) : 0.f));
      store_out(out, rh * DV + ch, o * invl * gate_of<bf16>(x, a, row, h0 + hh, ch), a);
    } else {
      part[(rh * a.nsplit + z) * DV + ch] = o;
      if (ch == 0) part_ml[rh * a.nsplit + z] = make_float2(m, l);
    }
  }
}

struct Call {
  const void* q;
  int ldq;
  const bf16* kcache;
  long long kss;
  const bf16* vcache;
  long long vss;
  const int* meta;
  const int* segs;
  int nseg;
  WindowExtras x;
  bf16* out;
  float* ws;
  int M;
  WindowArgs a;
  cudaStream_t stream;
};

template <int DK, int DV, int NQ> int prompt_as(const Call& c, int most = INT_MAX, int tiles = 0) {
  constexpr int smem = PromptShape<DK, DV, NQ>::SMEM;
  LIA_CUDA(cudaFuncSetAttribute(window_prompt_kernel<DK, DV, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const dim3 grid(c.a.H, tiles > 0 ? tiles : (c.M + BM - 1) / BM + (c.segs ? c.nseg - 1 : 0));     // at least as many tiles as the portions have
  lia_launch(window_prompt_kernel<DK, DV, NQ>, dim3(grid), dim3(128), smem, c.stream, c.q, c.ldq, c.kcache, c.kss, c.vcache, c.vss, c.meta, c.segs, c.nseg, most, c.x, c.out, c.M, c.a);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

template <int DK, int DV, int NQ> int decode_as(const Call& c) {
  const int smem = 4 * 8 * DV * (int)sizeof(float);
  float* part = c.ws;
  float2* part_ml = reinterpret_cast<float2*>(c.ws + (size_t)c.M * c.a.H * c.a.nsplit * DV);
  const dim3 grid((unsigned)(c.M * (c.a.H / c.a.HB)), c.a.nsplit);
  lia_launch(window_decode_kernel<DK, DV, NQ>, dim3(grid), dim3(128), smem, c.stream, c.q, c.ldq, c.kcache, c.kss, c.vcache, c.vss, c.meta, c.x, c.out, part, part_ml, c.a);
  LIA_LAUNCH_CHECK();
  if (c.a.nsplit > 1) return window_combine(part, part_ml, c.out, 0, c.M, c.x, c.a, c.stream);
  return LIA_OK;
}

// What lia_window_prompt_form returns: one kernel for all portions or, by their rows, both; above these bits, in 14 each, the tiles of either (0: not known)
enum { TCGEN05 = 2, MMA_SYNC = 3, BOTH = 4 };
constexpr int TILE_BITS = 14, TILE_MASK = (1 << TILE_BITS) - 1;

template <int DK, int DV> int run_as(const Call& c, int prompt) {
  if (prompt) {
    if constexpr (DK == 128 && DV == 128) {
      if (prompt == 1 || (!c.segs && prompt != MMA_SYNC)) prompt = lia_window_prompt_form(nullptr, c.segs ? c.nseg : 1, c.M, c.a.H, c.a.window, c.a.chunk, c.a.gate_mode == 2);      // (without segments there is one portion)
      const int kernels = prompt & 7, tc_tiles = prompt >> 3 & TILE_MASK, tiles = prompt >> (3 + TILE_BITS) & TILE_MASK;
      if (kernels != MMA_SYNC) {
        const int rc = window_prompt_tc(c.q, c.ldq, c.kcache, c.kss, c.vcache, c.vss, c.meta, c.segs, c.nseg, c.x, c.out, c.M, c.a, kernels == BOTH ? SHORT_ROWS + 1 : 1, tc_tiles, c.stream);
        if (rc != LIA_OK || kernels == TCGEN05) return rc;
      }
      const int most = kernels == BOTH ? SHORT_ROWS : INT_MAX;
      return c.a.q_f32 ? prompt_as<DK, DV, 3>(c, most, tiles) : prompt_as<DK, DV, 1>(c, most, tiles);
    } else {
      return c.a.q_f32 ? prompt_as<DK, DV, 3>(c) : prompt_as<DK, DV, 1>(c);
    }
  }
  return c.a.q_f32 ? decode_as<DK, DV, 3>(c) : decode_as<DK, DV, 1>(c);
}

bool head_sizes_ok(int dim, int vdim) { return (dim == 64 || dim == 128) && (vdim == 64 || vdim == 128 || vdim == 256); }

}  // namespace

// A tile of 128 rows has its SM to itself on tcgen05, however few of the rows are there; one of 64 on mma.sync shares it with two others.  So the first is ahead where tiles are few or histories
// long, the second with many portions of few rows.  What a step takes is estimated, in us, from the times of 1500 steps of 1 to 64 portions of 1 to 2048 rows behind 0 to 2000 positions, 8 to 32
// heads, both types of queries (tcgen05: 6.4 a tile and 1.1 for 64 keys; mma.sync: 1.2 a tile of throughput and, with up to 16, 32 or 64 rows, 0.76, 1.1 or 1.3 for 32 keys, of which one
// tile alone takes 2.75 and 1.8; a gate per channel 2.8 and 4.3 to 8.5 a tile): the kernel with the smaller estimate is the slower one by 3 % or more in 47 of them, by 13 and 22 % at most.
// us, mma.sync | tcgen05, 32 heads on 8 key heads, rows @ positions before them: 2 @ 0 5.5 | 8.4; 64 @ 256 25 | 14; 32 portions of 16 @ 0 17 | 58, @ 500 118 | 132, @ 1000 210 | 193; of 40 @ 0
// 29 | 62, @ 256 92 | 99, @ 500 153 | 136; of 96 @ 0 60 | 76, @ 64 92 | 86; of 128 @ 0 80 | 77.
// A portion of more than 128 rows is always tcgen05's, so that its bits do not depend on its company; a shorter one's may, as those of its projections do (128 rows and fewer in a step are
// multiplied another way).  Where portions are not known on the host, mma.sync has the steps of more tiles than SMs whose portions have 128 rows or fewer on average.
extern "C" int lia_window_prompt_form(const int* portions, int nseg, int M, int H, int window, int chunk, int gated) {
  if (nseg <= 0 || M <= 0 || H <= 0) return TCGEN05;
  const int sms = lia_sm_count();
  if (!portions) return nseg > 1 && M <= 128ll * nseg && ((M + 127ll) / 128 + nseg - 1) * H > sms ? MMA_SYNC : TCGEN05;
  WindowArgs a{};
  a.window = window > 0 ? window : 1 << 30;
  a.chunk = chunk;
  struct Sums {
    long long tiles = 0;
    double longest = 0, all = 0;
    void take(double alone, double shared) { ++tiles, longest = alone > longest ? alone : longest, all += shared; }
  } tc[2], mma[2];                                                 // of the long portions, of the short ones
  for (int i = 0; i < nseg; ++i) {
    const int pos = portions[4 * i + 1], rows = portions[4 * i + 3], is_short = rows <= SHORT_ROWS;
    auto keys = [&](int r, int of) { return pos + (r + of < rows ? r + of : rows) - first_key(a, pos + r); };
    for (int r = 0; r < rows; r += 128) {
      const double t = 6.4 + 1.1 * ((keys(r, 128) + 63) / 64) + (!gated ? 0 : rows - r <= 16 ? 0.6 : 2.8);
      tc[is_short].take(t, t);
    }
    for (int r = 0; r < rows && is_short; r += 64) {
      const int n = (keys(r, 64) + 31) / 32, here = rows - r;
      mma[1].take(2.75 + 1.8 * n + (!gated ? 0 : here <= 16 ? 4.5 : here <= 32 ? 6.5 : 8.5), 1.2 + (here <= 16 ? 0.76 : here <= 32 ? 1.1 : 1.3) * n + (!gated ? 0 : here <= 16 ? 4.3 : 5.3));
    }
  }
  auto tc_time = [&](long long tiles, double longest, double all) {
    if (tiles == 0) return 0.0;
    const long long items = tiles * H, waves = (items + sms - 1) / sms;
    const double shared = items > 4ll * sms ? all * H / sms : all / tiles * waves;
    return shared > longest ? shared : longest;
  };
  const double shared = mma[1].all * H / sms, both = shared < mma[1].longest ? mma[1].longest + 0.15 * shared : shared + 0.15 * mma[1].longest;
  const double one = tc_time(tc[0].tiles + tc[1].tiles, tc[0].longest > tc[1].longest ? tc[0].longest : tc[1].longest, tc[0].all + tc[1].all);
  if (mma[1].tiles == 0 || one <= tc_time(tc[0].tiles, tc[0].longest, tc[0].all) + both) return TCGEN05;
  if (tc[0].tiles == 0) return MMA_SYNC;
  return BOTH | (tc[0].tiles <= TILE_MASK && mma[1].tiles <= TILE_MASK ? (int)tc[0].tiles << 3 | (int)mma[1].tiles << (3 + TILE_BITS) : 0);
}

// 1 if the tensor-core kernels take bf16 caches of these head sizes, addresses and strides (elements); everything else is window_attn.cu's
extern "C" int lia_window_attn_mma_takes(const void* q, int ldq, int q_f32, const void* kcache, long long k_slot_stride, const void* vcache,
                                         long long v_slot_stride, const void* out, int H, int G, int v_div, int dim, int vdim) {
  const uintptr_t addr = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache) | reinterpret_cast<uintptr_t>(out);
  return head_sizes_ok(dim, vdim) && addr % 16 == 0 && ldq % (q_f32 ? 4 : 8) == 0 && k_slot_stride % 8 == 0 && v_slot_stride % 8 == 0 && H > 0 && G > 0 &&
         H % G == 0 && v_div > 0 && G % v_div == 0;
}

// The tensor-core form of lia_window_attn_masked for bf16 caches.  `prompt` (1, or what lia_window_prompt_form says): rows in portions `segs` [nseg][4] on the device (null: all rows are one
// portion that continues from meta[0]); otherwise every row by itself, its keys in nsplit ranges.
extern "C" int lia_window_attn_mma(const void* q, int ldq, int q_f32, const void* kcache, long long k_slot_stride, const void* vcache,
                                   long long v_slot_stride, const int* meta, const int* segs, int nseg, const float* temp, const float* slopes,
                                   const float* sink, const void* gate, int gate_mode, int ldg, void* out, int out_f32, float* workspace, int M, int H,
                                   int G, int v_div, int dim, int vdim, int window, int chunk, float scale, float softcap, int prompt, int nsplit,
                                   lia_stream_t stream_) {
  LIA_CHECK_ARG(q && kcache && vcache && meta && out && M > 0 && H <= 65535 && ldq >= H * dim && chunk >= 0, "lia_window_attn_mma: bad arguments");
  LIA_CHECK_ARG(lia_window_attn_mma_takes(q, ldq, q_f32, kcache, k_slot_stride, vcache, v_slot_stride, out, H, G, v_div, dim, vdim),
                "lia_window_attn_mma: heads of %d + %d channels, these addresses or strides are not for the tensor-core kernels", dim, vdim);
  LIA_CHECK_ARG(gate_mode >= 0 && gate_mode <= 2 && (gate_mode == 0) == (gate == nullptr) && (gate_mode != 2 || ldg >= H * vdim),
                "lia_window_attn_mma: bad output gate (mode %d, row stride %d)", gate_mode, ldg);
  LIA_CHECK_ARG(prompt >= 0 && (prompt & 7) <= BOTH && (prompt <= BOTH || (prompt & 7) == BOTH), "lia_window_attn_mma: no such form of prompts (%d)", prompt);
  LIA_CHECK_ARG(nsplit >= 1 && nsplit <= 64 && (nsplit == 1 || (workspace && prompt == 0)), "lia_window_attn_mma: bad number of key ranges (%d)", nsplit);
  LIA_CHECK_ARG(!prompt || (segs ? nseg > 0 && (M + BM - 1) / BM + nseg - 1 <= 65535 : (M + BM - 1) / BM <= 65535), "lia_window_attn_mma: bad portions");
  const int rep = H / G;
  int HB = rep < 8 ? rep : 8;
  while (rep % HB) --HB;
  WindowArgs a{H, G, dim, vdim, window > 0 ? window : 1 << 30, HB, 1, 1, nsplit, scale, softcap, q_f32, gate_mode, ldg};
  a.chunk = chunk;
  a.v_div = v_div;
  a.out_f32 = out_f32;
  const Call c{q, ldq, reinterpret_cast<const bf16*>(kcache), k_slot_stride, reinterpret_cast<const bf16*>(vcache), v_slot_stride, meta, segs, nseg,
               WindowExtras{temp, slopes, sink, gate}, reinterpret_cast<bf16*>(out), workspace, M, a, reinterpret_cast<cudaStream_t>(stream_)};
  if (dim == 64) {
    if (vdim == 64) return run_as<64, 64>(c, prompt);
    if (vdim == 128) return run_as<64, 128>(c, prompt);
    return run_as<64, 256>(c, prompt);
  }
  if (vdim == 64) return run_as<128, 64>(c, prompt);
  if (vdim == 128) return run_as<128, 128>(c, prompt);
  return run_as<128, 256>(c, prompt);
}
