// Window attention (window_attn.cu) of prompts on tcgen05, for bf16 caches with heads of 128 channels.  Nothing is held in fewer bits than on the CUDA cores: bf16 queries, keys and values
// enter as they are, fp32 queries and the softmax's weights as three bf16 parts (mma.cuh), scores and sums are fp32.
//
// One CTA per (128 rows of one portion, query head), 64 keys at a time; who does what: attn_sm100.cuh.
// Bound: the softmax's latencies and its some 25 instructions a score, two scores an instruction where they come in pairs: a block takes 2 x 2000 clocks of a group; the products
// (512 multiply-adds a score, 896 for fp32 queries) 1300 to 2400 of the tensor cores.  Loops over 32 scores with small bodies, for unrolled over 64 they miss the instruction cache.
//
// The tensor cores cut sums off below the 24th bit, so chains are short: a score has three accumulators of two or three instructions of high products each, the small parts of fp32 queries
// before them (what is cut off those is off a small sum); a block's weighted values are summed apart, small parts first, and added to the running sums in fp32.
// Sums that are not finite stay so to the end, where such rows are formed again key by key (window_attn_rows.cuh): a masked key's weight of 0 still meets its value.
// Waits are bounded: a CTA that gives up leaves NaN and counts itself (lia_moe_timeouts_seen()).
//
// 16 heads on 8 key heads of 128; on mma.sync -> here, us, and the error against 64 bits in 1e-7, means over 16 inputs: 2048 rows, window of 1024 and soft cap 136 (1.91) -> 66 (1.72), the whole history
// and fp32 queries 182 (2.32) -> 63 (1.62); 700 rows behind 300 89 (2.22) -> 29 (1.88); portions of 300, 250, 200 29 (1.35) -> 14 (1.26); 100 rows behind 2000 130 -> 50 (behind
// 1500 2.71 -> 2.05); four portions of 117, 100, 87, 73 14 -> 10, behind a gate per channel 23 -> 13.  Where mma.sync is the faster one: lia_window_prompt_form.
#include <limits.h>

#include "act.cuh"
#include "attn_sm100.cuh"
#include "window_attn_rows.cuh"

namespace {

constexpr int KEYS = 64, CH = 32;                                  // of a block; scores that a thread has at a time
constexpr int Q_BYTES = ROWS * D * 2, KV_BYTES = KEYS * D * 2;     // two slabs of 64 channels each, 128 bytes a row, 16-byte pieces turned by the row
struct Tail : AttnTail {
  uint64_t kv_full[4], kv_empty[4];
};
template <int NQ> __host__ __device__ constexpr int stages() { return NQ == 1 ? 4 : 3; }
template <int NQ> __host__ __device__ constexpr int smem_bytes() { return NQ * Q_BYTES + stages<NQ>() * 2 * KV_BYTES + (int)sizeof(Tail) + 1024; }

// finish_scores (window_attn_rows.cuh) two at a time; `far`: query position - key position of the first
__device__ __forceinline__ void finish_pairs(f32x2 (&s)[CH / 2], float mul, const WindowArgs& a, float slope, int far) {
#pragma unroll
  for (int i = 0; i < CH / 2; ++i) s[i] = mul2(s[i], both(mul));
  if (a.softcap > 0.f) {
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) {
      float x, y;
      unpack2(s[i], x, y);
      top = fmaxf(top, fmaxf(fabsf(x), fabsf(y)));
    }
    if (top <= 0.3f * a.softcap) {                                 // (a NaN stays one)
      const f32x2 inv = both(1.0f / a.softcap), cap = both(a.softcap), minus = both(-a.softcap);
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) {
        const f32x2 q = mul2(s[i], inv), b = fma2(fma2(q, minus, s[i]), inv, q), z = mul2(b, b);
        const f32x2 p = mul2(z, fma2(z, fma2(z, fma2(z, both(62.f / 2835.f), both(-17.f / 315.f)), both(2.f / 15.f)), both(-1.f / 3.f)));
        s[i] = mul2(cap, fma2(b, p, b));
      }
    } else {
#pragma unroll
      for (int i = 0; i < CH / 2; ++i) {
        float x, y;
        unpack2(s[i], x, y);
        s[i] = pack2(a.softcap * tanhf(x / a.softcap), a.softcap * tanhf(y / a.softcap));
      }
    }
  }
  if (slope != 0.f) {
#pragma unroll
    for (int i = 0; i < CH / 2; ++i) {
      float x, y;
      unpack2(s[i], x, y);
      s[i] = pack2(x - slope * (float)(far - 2 * i), y - slope * (float)(far - 2 * i - 1));
    }
  }
}

// A group's blocks s, s + 2, ... of n.  A thread's row is at position `pos` and sees the keys lo .. pos; its warp's first row is at wpos and sees keys from w_lo on, its last from w_all on; the
// first key is jb.  finish(pairs, j): what becomes of the sums of products with the keys j, j + 1, ...
template <class Finish>
__device__ __forceinline__ void softmax_blocks(AttnTail& sm, uint32_t tmem, int s, int n, int jb, int pos, int lo, int wpos, int w_lo, int w_all, const Finish& finish) {
  volatile int* dead = &sm.dead;
  const int w = group_warp(), lane = threadIdx.x & 31, r = w * 32 + lane;
  const uint32_t ts = tmem + s * GROUP + ((uint32_t)(w * 32) << 16);
#pragma unroll 1
  for (int it = s; it < n; it += 2) {
    const int j0 = jb + it * KEYS;
    if (!warp_wait(smem_u32(&sm.s_full[s]), (it >> 1) & 1, dead)) break;
    tcgen05_fence_after();
    const bool seen = j0 <= wpos + 31 && j0 + KEYS - 1 >= w_lo, partly = j0 + KEYS - 1 > wpos || j0 < w_all;         // by some row of the warp; not by every row, not every key
    float top = -INFINITY;
    if (seen) {
#pragma unroll 1
      for (int c = 0; c < KEYS; c += CH) {
        uint32_t u[3][CH];
#pragma unroll
        for (int k = 0; k < 3; ++k) tmem_ld32(ts + k * KEYS + c, u[k]);
        tmem_ld_wait();
        f32x2 sc[CH / 2];
#pragma unroll
        for (int i = 0; i < CH / 2; ++i) {
          f32x2 v[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) v[k] = pack2(__uint_as_float(u[k][2 * i]), __uint_as_float(u[k][2 * i + 1]));
          sc[i] = add2(add2(v[0], v[1]), v[2]);
        }
        finish(sc, j0 + c);
#pragma unroll
        for (int i = 0; i < CH / 2; ++i) {
          float x, y;
          unpack2(sc[i], x, y);
          u[0][2 * i] = __float_as_uint(x), u[0][2 * i + 1] = __float_as_uint(y);
        }
        if (partly) {
#pragma unroll
          for (int e = 0; e < CH; ++e)
            if (j0 + c + e > pos || j0 + c + e < lo) u[0][e] = 0xff800000u;
        }
        float t[4] = {top, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < CH; ++e) t[e & 3] = fmaxf(t[e & 3], __uint_as_float(u[0][e]));
        top = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3]));
        tmem_st32(ts + c, u[0]);
      }
      tmem_st_wait();
    }
    float before;
    if (!hand_over_top(sm, s, it, top, before)) break;
    const float from = top == -INFINITY ? 0.f : top;             // no key seen so far
    f32x2 sum[2] = {0ull, 0ull};
    if (seen) {
#pragma unroll 1
      for (int c = 0; c < KEYS; c += CH) {
        uint32_t u[CH], p[3][CH / 2];
        tmem_ld32(ts + c, u);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < CH / 2; ++i) {
          const f32x2 w = exp_pair(add2(pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1])), both(-from)));
          sum[i & 1] = add2(sum[i & 1], w);
          split_pair(w, p[0][i], p[1][i], p[2][i]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) tmem_st16(ts + WEIGHTS + k * 32 + c / 2, p[k]);
      }
    } else {
      const uint32_t none[16] = {};
#pragma unroll
      for (int c = 0; c < 96; c += 16) tmem_st16(ts + WEIGHTS + c, none);
    }
    float x, y;
    unpack2(add2(sum[0], sum[1]), x, y);
    sm.add[it & 3][r] = make_float2(expf(before - from), x + y);
    tmem_st_wait();
    tcgen05_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sm.p_full[s]));
  }
}

template <int NQ>
__global__ void __launch_bounds__(THREADS, 1) window_prompt_tc_kernel(const void* __restrict__ q, int ldq, const bf16* __restrict__ kcache, long long k_slot_stride,
                                                                      const bf16* __restrict__ vcache, long long v_slot_stride, const int* __restrict__ meta, const int* __restrict__ segs,
                                                                      int nseg, int least, WindowExtras x, bf16* __restrict__ out, int M, WindowArgs a, int* timeouts) {
  constexpr int ST = stages<NQ>();
  extern __shared__ uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u, ks = base + NQ * Q_BYTES;          // a stage: keys, values
  Tail& sm = *reinterpret_cast<Tail*>(raw + (base - smem_u32(raw)) + NQ * Q_BYTES + ST * 2 * KV_BYTES);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* dead = &sm.dead;
  if (tid == 0) {
    init_hand_overs(sm);
    for (int i = 0; i < ST; ++i) {
      mbar_init(smem_u32(&sm.kv_full[i]), LOADERS);
      mbar_init(smem_u32(&sm.kv_empty[i]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t tmem = take_tmem(sm, warp);
  pdl_launch_dependents();
  pdl_wait();
  int tile = gridDim.y - 1 - blockIdx.y, slot, pos0, row0, rows;
  if (segs == nullptr) {
    slot = meta[0]; pos0 = meta[1]; row0 = 0; rows = M;
    if (tile * ROWS >= rows) return give_tmem_back(tmem, warp);
  } else {
    const int found = portion_of<ROWS>(segs, nseg, tile, least, INT_MAX);
    if (found < 0) return give_tmem_back(tmem, warp);
    slot = segs[4 * found]; pos0 = segs[4 * found + 1]; row0 = segs[4 * found + 2]; rows = segs[4 * found + 3];
  }
  const int h = blockIdx.x, kg = h / (a.H / a.G), vg = kg / a.v_div, Gv = a.G / a.v_div;
  row0 += tile * ROWS;
  pos0 += tile * ROWS;
  rows = min(ROWS, rows - tile * ROWS);
  const size_t k_stride = (size_t)a.G * D, v_stride = (size_t)Gv * D;
  const float mul = a.scale * (x.temp ? x.temp[h] : 1.0f), slope = x.slopes ? x.slopes[h] : 0.f;
  auto by_itself = [&](size_t row, int slot_, int pos) {           // one row by one warp
    const PlainRow<D> y = plain_row<D, D, NQ>(q, row * ldq + (size_t)h * D, kcache + (size_t)slot_ * k_slot_stride + (size_t)kg * D, k_stride,
                                              vcache + (size_t)slot_ * v_slot_stride + (size_t)vg * D, v_stride, first_key(a, pos), pos, pos, mul, slope, a.softcap);
    const float invl = 1.0f / (y.l + (x.sink ? expf(x.sink[h] - y.m) : 0.f));
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      const int ch = lane + 32 * c;
      store_out(out, (row * a.H + h) * D + ch, y.o[c] * invl * gate_of<bf16>(x, a, row, h, ch), a);
    }
  };
  if (segs == nullptr) {                                           // what meta says counts: rows that do not continue one sequence go one by one
    bool run = true;
    if (tid < rows) run = meta[2 * (row0 + tid)] == slot && meta[2 * (row0 + tid) + 1] == pos0 + tid;
    if (!__syncthreads_and(run)) {
#pragma unroll 1
      for (int r = warp; r < rows; r += THREADS / 32) by_itself(row0 + r, meta[2 * (row0 + r)], meta[2 * (row0 + r) + 1]);
      return give_tmem_back(tmem, warp);
    }
  }
  slot = __shfl_sync(0xffffffffu, slot, 0), pos0 = __shfl_sync(0xffffffffu, pos0, 0), row0 = __shfl_sync(0xffffffffu, row0, 0), rows = __shfl_sync(0xffffffffu, rows, 0);      // known to be the same in all lanes
  const int pos_last = pos0 + rows - 1, jb = first_key(a, pos0), n = (pos_last - jb) / KEYS + 1;

  if (warp >= LOADER0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OTHER_REGS));
    if (warp < ISSUER) {
      const int piece = lane & 15;                                 // a piece of 16 bytes a lane and row, of keys and of values
      const bf16* kc = kcache + (size_t)slot * k_slot_stride + (size_t)kg * D + piece * 8;
      const bf16* vc = vcache + (size_t)slot * v_slot_stride + (size_t)vg * D + piece * 8;
      int under_way = -1;                                          // the block that was asked for last
      auto arrived = [&] {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.kv_full[under_way % ST]));
      };
#pragma unroll 1
      for (int it = 0; it < n; ++it) {
        const int st = it % ST, j0 = jb + it * KEYS;
        if (under_way >= 0 && !warp_test(smem_u32(&sm.kv_empty[st]), ((it / ST) & 1) ^ 1u)) {          // no place yet: first see the last one home
          cp_async_wait<0>();
          arrived();
          under_way = -1;
        }
        if (!warp_wait(smem_u32(&sm.kv_empty[st]), ((it / ST) & 1) ^ 1u, dead)) break;
        const uint32_t dst = ks + st * 2 * KV_BYTES + (piece >> 3) * (KV_BYTES / 2);
#pragma unroll 4
        for (int i = 2 * (warp - LOADER0) + (lane >> 4); i < KEYS; i += 2 * LOADERS) {
          const bool in = j0 + i <= pos_last;
          const size_t row = (size_t)(in ? j0 + i : pos_last);
          const uint32_t at = dst + i * 128 + (((piece & 7) ^ (i & 7)) << 4);
          cp_async16(at, kc + row * k_stride, in ? 16 : 0);        // rows behind the last are zero
          cp_async16(at + KV_BYTES, vc + row * v_stride, in ? 16 : 0);
        }
        cp_async_commit();
        if (under_way >= 0) {
          cp_async_wait<1>();
          arrived();
        }
        under_way = it;
      }
      cp_async_wait<0>();
      if (under_way >= 0) arrived();
    } else {
      const uint32_t one = elect_one();
      constexpr uint32_t idesc_s = make_idesc(ROWS, KEYS);
      // (from loops: unrolled, these instructions would not stay in the instruction cache beside the other warps' code)
      const uint64_t q_desc = make_smem_desc(base), k_desc = make_smem_desc(ks), v_desc = make_smem_desc_mn(ks + KV_BYTES, KV_BYTES / 2);
      auto scores = [&](int it) {
        const uint64_t kt = k_desc + (uint32_t)(it % ST) * (2 * KV_BYTES >> 4);
        const uint32_t d = tmem + (it & 1) * GROUP;
#pragma unroll 1
        for (int part = NQ - 1; part >= 0; --part) {               // small parts first; the accumulators in turn, so that no instruction waits for the one before it
          uint64_t qa = q_desc + (uint32_t)part * (Q_BYTES >> 4), kb = kt;
          uint32_t to = d;
#pragma unroll 1
          for (int slab = 0; slab < 2; ++slab, qa += Q_BYTES >> 5, kb += KV_BYTES >> 5)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              mma_if(one, to, qa + 2 * k, kb + 2 * k, idesc_s, part < NQ - 1 || slab > 0 || k == 3);
              to = to == d + 2 * KEYS ? d : to + KEYS;
            }
        }
        commit_if(one, smem_u32(&sm.s_full[it & 1]));
      };
      bool alive = warp_wait(smem_u32(&sm.q_full), 0u, dead);
      for (int it = 0; alive && it < 2 && it < n; ++it) {
        alive = warp_wait(smem_u32(&sm.kv_full[it]), 0u, dead);
        tcgen05_fence_after();
        if (alive) scores(it);
      }
#pragma unroll 1
      for (int it = 0; alive && it < n; ++it) {
        const int s = it & 1;
        if (!(alive = warp_wait(smem_u32(&sm.p_full[s]), (it >> 1) & 1, dead))) break;
        tcgen05_fence_after();
        const uint64_t vb = v_desc + (uint32_t)(it % ST) * (2 * KV_BYTES >> 4);
#pragma unroll 1
        for (int part = 2; part >= 0; --part) issue_values<KEYS>(one, tmem, s, part, vb, part == 2);
        commit_if(one, smem_u32(&sm.kv_empty[it % ST]));
        commit_if(one, smem_u32(&sm.o_full));
        if (it + 2 < n) {
          if (!(alive = warp_wait(smem_u32(&sm.kv_full[(it + 2) % ST]), ((it + 2) / ST) & 1, dead))) break;
          tcgen05_fence_after();
          scores(it + 2);
        }
      }
    }
    __syncwarp();
  } else if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGS));
    {
      const int c = tid & 15;                                      // 8 channels of every 16th row, all asked for at once
      uint4 v[8][NQ == 1 ? 1 : 2];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid >> 4) + i * 16;
        const size_t at = (size_t)(row0 + r) * ldq + (size_t)h * D + c * 8;
#pragma unroll
        for (int k = 0; k < (NQ == 1 ? 1 : 2); ++k)
          v[i][k] = r < rows ? reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(q) + at * (NQ == 1 ? 2 : 4))[k] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (tid >> 4) + i * 16;
        uint32_t part[NQ][4];
        if constexpr (NQ == 1) {
          part[0][0] = v[i][0].x; part[0][1] = v[i][0].y; part[0][2] = v[i][0].z; part[0][3] = v[i][0].w;
        } else {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            split3(__uint_as_float(v[i][k].x), __uint_as_float(v[i][k].y), part[0][2 * k], part[1][2 * k], part[2][2 * k]);
            split3(__uint_as_float(v[i][k].z), __uint_as_float(v[i][k].w), part[0][2 * k + 1], part[1][2 * k + 1], part[2][2 * k + 1]);
          }
        }
#pragma unroll
        for (int s = 0; s < NQ; ++s)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(base + s * Q_BYTES + (c >> 3) * (Q_BYTES / 2) + r * 128 + (((c & 7) ^ (r & 7)) << 4)), "r"(part[s][0]), "r"(part[s][1]),
                       "r"(part[s][2]), "r"(part[s][3]) : "memory");
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sm.q_full));

    const int s = warp >> 2, r = (warp & 3) * 32 + lane, pos = pos0 + r, wpos = pos0 + (warp & 3) * 32, lo = first_key(a, pos);
    const int w_lo = first_key(a, wpos), w_all = first_key(a, wpos + 31);
    softmax_blocks(sm, tmem, s, n, jb, pos, lo, wpos, w_lo, w_all, [&](f32x2 (&sc)[CH / 2], int j) { finish_pairs(sc, mul, a, slope, pos - j); });
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SUM_REGS));
    const int r0 = (warp & 3) * 32;
    f32x2 O[D / 2];
    double l;
    const bool alive = sum_blocks(sm, tmem, n, O, l);
    const float inv = alive ? 1.0f / ((float)l + (x.sink ? expf(x.sink[h] - sm.top[(n - 1) & 1][r0 + lane]) : 0.f)) : NAN;
    // Every product is done: the sums' way out takes the keys' and values' place, the gates, before their sigmoid, the queries'.  By way of shared memory they are under way while the sums are written,
    // and a loop of four rows is enough; eight rows' in registers, with the compiler's division, took a tile 10 us for 2.8 (mma.sync: 4.5 to 8.5).
    uint8_t* gates = raw + (base - smem_u32(raw)) + (warp & 3) * (32 * D * 2);
    float head_gate = 0.f;
    if (a.gate_mode == 1 && r0 + lane < rows) head_gate = reinterpret_cast<const float*>(x.gate)[(size_t)(row0 + r0 + lane) * a.H + h];
    if (a.gate_mode == 2) {
      const unsigned short* g = reinterpret_cast<const unsigned short*>(x.gate) + (size_t)(row0 + r0) * a.ldg + (size_t)h * D + lane * 4;
      const int n = min(32, rows - r0);
      if ((reinterpret_cast<uintptr_t>(x.gate) | (uintptr_t)(a.ldg * 2)) % 8 == 0) {
#pragma unroll 4
        for (int i = 0; i < n; ++i) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(gates) + i * (D * 2) + lane * 8), "l"(g + (size_t)i * a.ldg) : "memory");
      } else {
#pragma unroll 1
        for (int i = 0; i < n; ++i, g += a.ldg) reinterpret_cast<uint2*>(gates)[i * 32 + lane] = make_uint2(g[0] | (uint32_t)g[1] << 16, g[2] | (uint32_t)g[3] << 16);
      }
      cp_async_commit();
    }
    auto gate = [&](int i, float4& y) {
      float4 g;
      if (a.gate_mode == 1) {
        g.x = g.y = g.z = g.w = __shfl_sync(0xffffffffu, head_gate, i);
      } else {
        const uint2 u = reinterpret_cast<const uint2*>(gates)[i * 32 + lane];
        unpack_bf16x2(u.x, g.x, g.y);
        unpack_bf16x2(u.y, g.z, g.w);
        g = make_float4(over(1.0f, 1.0f + expf(-g.x)), over(1.0f, 1.0f + expf(-g.y)), over(1.0f, 1.0f + expf(-g.z)), over(1.0f, 1.0f + expf(-g.w)));
      }
      y = make_float4(y.x * g.x, y.y * g.y, y.z * g.z, y.w * g.w);
    };
    const unsigned again = rows_out(raw + (ks - smem_u32(raw)) + (warp & 3) * (32 * D * 4), O, inv, alive, rows - r0, a.gate_mode != 0, gate, [&](int i, float4 y) {
      const size_t at = ((size_t)(row0 + r0 + i) * a.H + h) * D + lane * 4;
      if (a.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + at) = y;
      else *reinterpret_cast<uint2*>(out + at) = make_uint2(pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
    });
    if (again) {
#pragma unroll 1
      for (int i = 0; i < 32; ++i)
        if ((again >> i) & 1u) by_itself(row0 + r0 + i, slot, pos0 + r0 + i);
    }
  }
  leave(sm, tmem, warp, timeouts, [] {});                          // (each loading thread has waited for its own)
}

template <int NQ>
int launch(const void* q, int ldq, const bf16* kcache, long long kss, const bf16* vcache, long long vss, const int* meta, const int* segs, int nseg, const WindowExtras& x, bf16* out, int M,
           const WindowArgs& a, int least, int tiles, cudaStream_t stream) {
  constexpr int smem = smem_bytes<NQ>();
  static_assert(smem <= 232448, "shared memory budget exceeded");
  LIA_CUDA(cudaFuncSetAttribute(window_prompt_tc_kernel<NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  static const bool split_fits = registers_suffice(window_prompt_tc_kernel<NQ>);
  LIA_CHECK_ARG(split_fits, "lia_window_attn_mma: built with another number of registers");
  int* timeouts = lia_timeout_word();
  LIA_CHECK_ARG(timeouts != nullptr, "lia_window_attn_mma: no host memory for the count of timeouts");
  const dim3 grid(a.H, tiles > 0 ? tiles : (M + ROWS - 1) / ROWS + (segs ? nseg - 1 : 0));   // at least as many tiles as the portions have
  lia_launch(window_prompt_tc_kernel<NQ>, grid, dim3(THREADS), smem, stream, q, ldq, kcache, kss, vcache, vss, meta, segs, nseg, least, x, out, M, a, timeouts);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

}  // namespace

// The prompt form of lia_window_attn_mma for heads of 128 + 128 channels, for the portions of `least` rows and more; `tiles`: of 128 rows, that these have (0: not known)
int window_prompt_tc(const void* q, int ldq, const bf16* kcache, long long kss, const bf16* vcache, long long vss, const int* meta, const int* segs, int nseg, const WindowExtras& x, bf16* out,
                     int M, const WindowArgs& a, int least, int tiles, cudaStream_t stream) {
  return a.q_f32 ? launch<3>(q, ldq, kcache, kss, vcache, vss, meta, segs, nseg, x, out, M, a, least, tiles, stream)
                 : launch<1>(q, ldq, kcache, kss, vcache, vss, meta, segs, nseg, x, out, M, a, least, tiles, stream);
}
