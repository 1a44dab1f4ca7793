// Latent portions over expanded keys and values (latent_attn_mma.cu) on tcgen05, for heads of 128 + 64 channels.  Keys and values are three bf16 parts of their fp32 sums, as are the rotated query
// parts and the softmax's weights (mma.cuh); with bf16 queries and bf16 rotated keys a score is three products of each part, a weighted value six (of the nine).
//
// One CTA per (128 rows of a portion, head), 32 keys at a time; who does what: attn_sm100.cuh.  Bound: the tensor cores and the warp that feeds them, 40 instructions a block of 47 (scores) and 62
// (values) clocks each and 600 clocks between them.  A block's parts are 52 KB from L2, by TMA where they are the workspace's (by cp.async of three warps: 7900 clocks per 64 keys, 4100 by TMA);
// shared memory holds two blocks.
//
// The tensor cores cut sums off below the 24th bit, so chains are short: a score has six accumulators of two instructions of high products each, the small products before them (the keys' two
// lower parts side by side in one instruction).  It stays unscaled until it is taken off the maximum, so that the scale's rounding is that of a small number.  With 64 keys and three accumulators
// of four high products (83 us instead of 104 of the first example below) outputs were off by 1.06 to 1.18 times what mma.sync gave, with 48 and four by 1.03 to 1.05.  A block's weighted values
// go from small to large and are added to the running sums in fp32.
// Sums that are not finite stay so to the end, where such rows are formed again key by key: a masked key's weight of 0 still meets its value.
// Waits are bounded: a CTA that gives up leaves NaN and counts itself (lia_moe_timeouts_seen()).
//
// Latents of 512, with their expansion (latent_expand_sm100.cu); on mma.sync -> here, us, and the error against 64 bits in 1e-7, means over 16 inputs: 2048 rows, 16 heads 413 (1.97) -> 130 (1.83); 700
// rows behind 300, 32 heads 250 (2.22) -> 96 (2.08); portions of 300, 250 and 200, 16 heads 88 (1.75) -> 36 (1.60); 64 rows 28 (1.55) -> 14 (1.41); 100 rows behind 1500, 32 heads 376 (2.30) -> 122
// (2.22), 8 heads 210 (2.30) -> 89 (2.23).
#include "attn_sm100.cuh"
#include "latent_attn_rows.cuh"

namespace {

constexpr int DN = 128, DR = 64, KEYS = 32, ACCS = 6, CH = 16;
constexpr int SLAB = KEYS * 128;                                   // of 64 channels
// in shared memory, bytes from the first; rows of 128 bytes in slabs of 64 channels, their 16-byte pieces turned by the row; the keys and values of two blocks, STAGE apart
constexpr int QN = 0, QR = QN + ROWS * DN * 2, K_SMALL = QR + 3 * ROWS * DR * 2, K_HIGH = K_SMALL + 4 * SLAB, K_ROT = K_HIGH + 2 * SLAB, V_LOW = K_ROT + SLAB, V_MID = V_LOW + 2 * SLAB,
              V_HIGH = V_MID + 2 * SLAB, STAGE = V_HIGH + 2 * SLAB - K_SMALL, TAIL = K_SMALL + 2 * STAGE;
struct Tail : AttnTail {
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  int issued[2];                                                   // blocks of keys, of values that were asked for by TMA
};
constexpr int SMEM = TAIL + (int)sizeof(Tail) + 1024;
static_assert(SMEM <= 232448 && TAIL - K_SMALL >= 4 * 32 * D * 4, "shared memory budget exceeded, or no place for the sums' way out");

// The rotated parts of the keys j0 .. j0 + KEYS - 1, by one warp, a piece of 16 bytes a lane and row, turned by the row; rows behind `last` as zeros
__device__ __forceinline__ void fetch_rotated(uint32_t dst, const bf16* rows, long long stride, int j0, int last) {
  const int lane = threadIdx.x & 31, piece = lane & 7;
#pragma unroll 4
  for (int i = lane >> 3; i < KEYS; i += 4) {
    const bool in = j0 + i <= last;
    cp_async16(dst + i * 128 + ((piece ^ (i & 7)) << 4), rows + (size_t)(in ? j0 + i : last) * stride + piece * 8, in ? 16 : 0);
  }
}

__global__ void __launch_bounds__(THREADS, 1) latent_expanded_tc_kernel(const __grid_constant__ ExpandedArgs a, const __grid_constant__ CUtensorMap map, int* timeouts) {
  extern __shared__ uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
  uint8_t* gen = raw + (base - smem_u32(raw));
  Tail& sm = *reinterpret_cast<Tail*>(gen + TAIL);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* dead = &sm.dead;
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map) : "memory");
    init_hand_overs(sm);
    for (int i = 0; i < 2; ++i) {
      sm.issued[i] = 0;
      mbar_init(smem_u32(&sm.k_full[i]), 2);
      mbar_init(smem_u32(&sm.v_full[i]), 1);
      mbar_init(smem_u32(&sm.k_empty[i]), 1);
      mbar_init(smem_u32(&sm.v_empty[i]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t tmem = take_tmem(sm, warp);
  pdl_launch_dependents();
  const int h = a.h0 + blockIdx.x, tile = gridDim.y - 1 - blockIdx.y;            // a portion's longest histories start first
  int ip = 0;
  while (ip + 1 < a.np && tile >= a.p[ip + 1].tile0) ++ip;
  const Portion& pt = a.p[ip];
  const int skip = (tile - pt.tile0) * ROWS, row0 = pt.row0 + skip;
  const int rows = min(ROWS, pt.n - skip), pos0 = pt.pos0 + skip, pos_last = pos0 + rows - 1;
  const int jb = max(0, pos0 - a.window + 1), n = (pos_last - jb) / KEYS + 1;
  const size_t key_stride = (size_t)a.nh * 6 * DN;
  const bf16* keys = a.parts + (size_t)pt.part0 * key_stride + (size_t)blockIdx.x * 3 * DN;
  const bf16* vals = keys + (size_t)a.nh * 3 * DN;
  const bf16* key_rot = pt.kr;
  // a weight is exp(unit (score sign - its maximum)); a scale near 0 goes to the scores
  const bool small_scale = fabsf(a.scale) < 1e-6f;
  const float sign = small_scale ? a.scale : a.scale < 0.f ? -1.f : 1.f, unit = small_scale ? 1.f : fabsf(a.scale);
  pdl_wait();

  if (warp >= LOADER0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OTHER_REGS));
    if (warp < ISSUER) {
      if (warp == LOADER0 + 1) {                                   // rotated key parts, from the cache
#pragma unroll 1
        for (int it = 0; it < n && warp_wait(smem_u32(&sm.k_empty[it & 1]), ((it >> 1) & 1) ^ 1u, dead); ++it) {
          fetch_rotated(base + K_ROT + (it & 1) * STAGE, key_rot, a.kr_stride, jb + it * KEYS, pos_last);
          cp_async_commit();
          cp_async_wait<0>();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sm.k_full[it & 1]));
        }
      } else {
        // keys (warp 12) and values (warp 14), the parts of a head side by side in a row: rows of 64 columns.  Rows behind the last are the next portion's, or zeros: no row sees them.
        const uint32_t one = elect_one();
        const bool of_keys = warp == LOADER0;
        const int col = (of_keys ? 0 : a.nh * 3 * DN) + blockIdx.x * 3 * DN, row = pt.part0 + jb;
#pragma unroll 1
        for (int it = 0; it < n; ++it) {
          const uint32_t full = smem_u32(of_keys ? &sm.k_full[it & 1] : &sm.v_full[it & 1]), empty = smem_u32(of_keys ? &sm.k_empty[it & 1] : &sm.v_empty[it & 1]);
          if (!warp_wait(empty, ((it >> 1) & 1) ^ 1u, dead)) break;
          if (!one) continue;
          sm.issued[of_keys ? 0 : 1] = it + 1;
          mbar_expect_tx(full, 6 * SLAB);
#pragma unroll
          for (int part = 2; part >= 0; --part) {
            const uint32_t at = base + (it & 1) * STAGE + (of_keys ? part == 0 ? K_HIGH : K_SMALL + (part - 1) * SLAB : part == 0 ? V_HIGH : part == 1 ? V_MID : V_LOW);
            const uint32_t slab = of_keys && part > 0 ? 2 * SLAB : SLAB;
#pragma unroll
            for (int k = 0; k < 2; ++k) tma_load_2d(at + k * slab, &map, col + part * DN + k * 64, row + it * KEYS, full);
          }
        }
      }
    } else {
      const uint32_t one = elect_one();
      constexpr uint32_t idesc1 = make_idesc(ROWS, KEYS), idesc2 = make_idesc(ROWS, 2 * KEYS);
      const uint64_t qn = make_smem_desc(base + QN), qr = make_smem_desc(base + QR), small = make_smem_desc(base + K_SMALL), high = make_smem_desc(base + K_HIGH), rot = make_smem_desc(base + K_ROT),
                     low = make_smem_desc_mn(base + V_LOW, SLAB), mid = make_smem_desc_mn(base + V_MID, SLAB), top = make_smem_desc_mn(base + V_HIGH, SLAB);
      // (from loops: unrolled, these instructions would not stay in the instruction cache beside the other warps' code)
      auto scores = [&](int it) {
        const uint32_t d = tmem + (it & 1) * GROUP;
        const uint64_t st = (uint64_t)((it & 1) * (STAGE >> 4));
        if (!warp_wait(smem_u32(&sm.k_full[it & 1]), (it >> 1) & 1, dead)) return false;
        tcgen05_fence_after();
#pragma unroll 1
        for (int slab = 0; slab < 2; ++slab)
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_if(one, d, qn + slab * (ROWS * 128 >> 4) + 2 * k, small + st + slab * (2 * SLAB >> 4) + 2 * k, idesc2, slab > 0 || k > 0);
#pragma unroll 1
        for (int part = 2; part >= 1; --part)
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_if(one, d + 2 * KEYS, qr + part * (ROWS * 128 >> 4) + 2 * k, rot + st + 2 * k, idesc1, part < 2 || k > 0);
        uint32_t to = d;                                           // the accumulators in turn, two instructions each; the third slab is the rotated part
#pragma unroll 1
        for (int slab = 0; slab < 3; ++slab) {
          const uint64_t qa = slab < 2 ? qn + slab * (ROWS * 128 >> 4) : qr, kb = st + (slab < 2 ? high + slab * (SLAB >> 4) : rot);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            mma_if(one, to, qa + 2 * k, kb + 2 * k, idesc1, slab == 0 ? k < 3 : slab == 2 || k > 1);
            to = to == d + (ACCS - 1) * KEYS ? d : to + KEYS;
          }
        }
        commit_if(one, smem_u32(&sm.s_full[it & 1]));
        commit_if(one, smem_u32(&sm.k_empty[it & 1]));
        return true;
      };
      bool alive = warp_wait(smem_u32(&sm.q_full), 0u, dead);
      for (int it = 0; alive && it < 2 && it < n; ++it) alive = scores(it);
#pragma unroll 1
      for (int it = 0; alive && it < n; ++it) {
        const int s = it & 1;
        const uint64_t st = (uint64_t)(s * (STAGE >> 4));
        if (!(alive = warp_wait(smem_u32(&sm.v_full[s]), (it >> 1) & 1, dead) && warp_wait(smem_u32(&sm.p_full[s]), (it >> 1) & 1, dead))) break;
        tcgen05_fence_after();
#pragma unroll 1
        for (int i = 0; i < 6; ++i) {                              // high x low, mid x mid, low x high, high x mid, mid x high, high x high
          const int part = (0x010210 >> (4 * i)) & 15;
          issue_values<KEYS>(one, tmem, s, part, st + (i == 0 ? low : i == 1 || i == 3 ? mid : top), i == 0);
        }
        commit_if(one, smem_u32(&sm.o_full));
        commit_if(one, smem_u32(&sm.v_empty[s]));
        if (it + 2 < n) alive = scores(it + 2);
      }
    }
    __syncwarp();
  } else if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGS));
    {
      uint4 v[8], u[4][2];                                         // 8 channels of every 16th row, 8 rotated ones of every 32nd, all asked for at once
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid >> 4) + i * 16;
        v[i] = r < rows ? *reinterpret_cast<const uint4*>(a.q + (size_t)(row0 + r) * a.ldq + (size_t)h * (DN + DR) + (tid & 15) * 8) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (tid >> 3) + i * 32;
        const uint4* src = reinterpret_cast<const uint4*>(a.qr + ((size_t)(row0 + r) * a.H + h) * a.qr_stride + (tid & 7) * 8);
#pragma unroll
        for (int k = 0; k < 2; ++k) u[i][k] = r < rows ? src[k] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid >> 4) + i * 16, c = tid & 15;
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(base + QN + (c >> 3) * (ROWS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)), "r"(v[i].x), "r"(v[i].y), "r"(v[i].z), "r"(v[i].w) : "memory");
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (tid >> 3) + i * 32, c = tid & 7;
        uint32_t p[3][4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          split3(__uint_as_float(u[i][k].x), __uint_as_float(u[i][k].y), p[0][2 * k], p[1][2 * k], p[2][2 * k]);
          split3(__uint_as_float(u[i][k].z), __uint_as_float(u[i][k].w), p[0][2 * k + 1], p[1][2 * k + 1], p[2][2 * k + 1]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(base + QR + k * (ROWS * 128) + r * 128 + ((c ^ (r & 7)) << 4)), "r"(p[k][0]), "r"(p[k][1]), "r"(p[k][2]), "r"(p[k][3]) : "memory");
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sm.q_full));
    const int s = warp >> 2, wpos = pos0 + (warp & 3) * 32, pos = wpos + lane, lo = pos - a.window + 1;
    const uint32_t ts = tmem + s * GROUP + ((uint32_t)((warp & 3) * 32) << 16);
    const double c = (double)unit * 1.4426950408889634;
    const float c_high = (float)c, c_rest = (float)(c - (double)c_high), least = -150.f / unit;
#pragma unroll 1
    for (int it = s; it < n; it += 2) {
      const int j0 = jb + it * KEYS;
      if (!warp_wait(smem_u32(&sm.s_full[s]), (it >> 1) & 1, dead)) break;
      tcgen05_fence_after();
      const bool seen = j0 <= wpos + 31 && j0 + KEYS - 1 >= wpos - a.window + 1, partly = j0 + KEYS - 1 > wpos || j0 < wpos + 31 - a.window + 1;       // by some row of the warp; not by every row, not every key
      float top = -INFINITY;
      if (seen) {
#pragma unroll 1
        for (int c = 0; c < KEYS; c += CH) {
          uint32_t u[ACCS][CH];
#pragma unroll
          for (int k = 0; k < ACCS; ++k) tmem_ld16(ts + k * KEYS + c, u[k]);
          tmem_ld_wait();
          float t[2] = {top, -INFINITY};
#pragma unroll
          for (int i = 0; i < CH / 2; ++i) {
            f32x2 v[ACCS];
#pragma unroll
            for (int k = 0; k < ACCS; ++k) v[k] = pack2(__uint_as_float(u[k][2 * i]), __uint_as_float(u[k][2 * i + 1]));
            float x, y;
            unpack2(mul2(add2(add2(add2(v[0], v[1]), add2(v[2], v[3])), add2(v[4], v[5])), both(sign)), x, y);
            if (partly) {
              const int j = j0 + c + 2 * i;
              if (j > pos || j < lo) x = -INFINITY;
              if (j + 1 > pos || j + 1 < lo) y = -INFINITY;
            }
            t[i & 1] = fmaxf(t[i & 1], fmaxf(x, y));
            u[0][2 * i] = __float_as_uint(x);
            u[0][2 * i + 1] = __float_as_uint(y);
          }
          top = fmaxf(t[0], t[1]);
          tmem_st16(ts + c, u[0]);
        }
        tmem_st_wait();
      }
      float before;
      if (!hand_over_top(sm, s, it, top, before)) break;
      const float from = top == -INFINITY ? 0.f : top;             // no key seen so far
      f32x2 sum[2] = {0ull, 0ull};
      uint32_t u[KEYS], p[3][KEYS / 2] = {};
      if (seen) {
        tmem_ld32(ts, u);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < KEYS / 2; ++i) {
          const f32x2 w = pow2_pair(add2(pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1])), both(-from)), c_high, c_rest, least);
          sum[i & 1] = add2(sum[i & 1], w);
          split_pair(w, p[0][i], p[1][i], p[2][i]);
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) tmem_st16(ts + WEIGHTS + k * (KEYS / 2), p[k]);
      float x, y;
      unpack2(add2(sum[0], sum[1]), x, y);
      sm.add[it & 3][(warp & 3) * 32 + lane] = make_float2(expf((before - from) * unit), x + y);
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.p_full[s]));
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SUM_REGS));
    const int r0 = (warp & 3) * 32;
    f32x2 O[D / 2];
    double l;
    const bool alive = sum_blocks(sm, tmem, n, O, l);
    // gate over the softmax's denominator, the sink among its terms: everything relative to the larger of maximum and sink
    auto factor = [&](size_t row, float m, float l) {
      const float f = a.gate ? a.gate[row * a.H + h] : 1.0f;
      if (a.sink == nullptr) return f / l;
      const float top = fmaxf(m, a.sink[h]), e = expf(m - top);
      return f * (e / (l * e + expf(a.sink[h] - top)));
    };
    const float inv = !alive ? NAN : r0 + lane < rows ? factor(row0 + r0 + lane, sm.top[(n - 1) & 1][r0 + lane] * unit, (float)l) : 0.f;
    // (the keys' and values' place: every product is done)
    const unsigned again = rows_out(gen + K_SMALL + (warp & 3) * (32 * D * 4), O, inv, alive, rows - r0, false, [](int, float4&) {}, [&](int i, float4 y) {
      const size_t at = ((size_t)(row0 + r0 + i) * a.H + h) * DN + lane * 4;
      if (a.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + at) = y;
      else *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(a.out) + at) = make_uint2(pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
    });
    if (again) {
#pragma unroll 1
      for (int i = 0; i < 32; ++i) {
        if (!((again >> i) & 1u)) continue;
        const size_t row = row0 + r0 + i;
        const int pos = pos0 + r0 + i;
        const PlainRow<DN> y = plain_row<DN, DR>(a.q + row * a.ldq + (size_t)h * (DN + DR), a.qr + (row * a.H + h) * a.qr_stride, keys, vals, key_stride, key_rot, a.kr_stride,
                                                 max(0, pos - a.window + 1), pos, a.scale);
        const float f = factor(row, y.m, y.l);
#pragma unroll
        for (int c = 0; c < DN / 32; ++c) {
          const size_t at = (row * a.H + h) * DN + lane + 32 * c;
          if (a.out_f32) reinterpret_cast<float*>(a.out)[at] = y.o[c] * f;
          else reinterpret_cast<bf16*>(a.out)[at] = __float2bfloat16_rn(y.o[c] * f);
        }
      }
    }
  }
  leave(sm, tmem, warp, timeouts, [&] {
    for (int i = 0; i < 2; ++i)
      for (int t = max(0, sm.issued[i] - 2); t < sm.issued[i]; ++t) wait_in_flight(smem_u32(i ? &sm.v_full[t & 1] : &sm.k_full[t & 1]), (t >> 1) & 1);
  });
}

}  // namespace

// `tiles`: of 128 rows, of all portions; `latents`: expanded rows
int latent_expanded_tc(const ExpandedArgs& a, int tiles, long long latents, cudaStream_t stream) {
  LIA_CUDA(cudaFuncSetAttribute(latent_expanded_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
  static const bool split_fits = registers_suffice(latent_expanded_tc_kernel);
  LIA_CHECK_ARG(split_fits, "lia_latent_attn_expanded: built with another number of registers");
  int* timeouts = lia_timeout_word();
  LIA_CHECK_ARG(timeouts != nullptr, "lia_latent_attn_expanded: no host memory for the count of timeouts");
  CUtensorMap map;
  const int rc = lia_make_tmap_2d(&map, a.parts, (uint64_t)latents, (uint64_t)a.nh * 6 * DN, (uint64_t)a.nh * 6 * DN, KEYS);
  if (rc != LIA_OK) return rc;
  lia_launch(latent_expanded_tc_kernel, dim3(a.nh, tiles), dim3(THREADS), SMEM, stream, a, map, timeouts);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}
