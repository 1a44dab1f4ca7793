// What the prompt kernels of attention on tcgen05 share (window_attn_sm100.cu, latent_attn_sm100.cu): a CTA of 16 warps has 128 rows of one head and takes their keys in blocks of KEYS.
//   warps 0-3, 4-7   two groups that take the blocks in turn (softmax_blocks); a thread owns one row, which is one lane of TMEM
//   warps 8-11       the running sums, a thread a row (sum_blocks, rows_out)
//   warps 12-14      loads;  warp 15: the products
// TMEM, 512 columns: group s has its scores at GROUP s, in three accumulators of 64 columns or six of 32, whose sum is the score; in their place come the weights, in three bf16 parts (the A
// operand of the products with the values), at WEIGHTS.  The weighted values of a block, of either group, lie at SUMS.
// The order of a block's hand-overs: s_full (scores are there), m_full (the running maximum; a warp's rows go to the same warp of the other group), p_full (weights are there, and the weighted
// values of the block before are added up: their place is free), o_full (weighted values).  A group's next scores are issued behind the products with its weights, in whose place they come.  Few
// barriers, for one that is long complete still costs the warp that issues 150 clocks.
#pragma once
#include <type_traits>

#include "mma.cuh"
#include "umma.cuh"

int* lia_timeout_word();                                           // moe_sm100.cu

namespace {

constexpr int ROWS = 128, D = 128;                                 // D: value columns of a head
constexpr int THREADS = 512, LOADERS = 3, LOADER0 = 12, ISSUER = 15;
constexpr int SOFTMAX_REGS = 144, SUM_REGS = 184, OTHER_REGS = 40; // of a thread, by what its four warps do (setmaxnreg: multiples of 8)
constexpr uint32_t GROUP = 192, WEIGHTS = 64, SUMS = 384;

struct AttnTail {
  float top[2][ROWS];                                              // the running maximum after a block
  float2 add[4][ROWS];                                             // of a block: what the sums before it count for, the sum of its weights
  uint64_t q_full, s_full[2], p_full[2], m_full[2][4], o_full, drain;
  uint32_t tmem;
  int dead;
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 both(float x) { return pack2(x, x); }

// 2^(x (c + c_rest)) for x <= 0: the power of the rounded product, corrected to first order by what the rounding of the product and of the factor left out.  x below `least` count as that, so
// that no infinity less itself comes of them; a NaN stays one.  (Results below 2^-126 are kept, as expf keeps them: cut off to 0 they are three instructions less a weight, 54 us for 56 of window
// attention's 2048 rows and 16 heads.  Found by the least score of a block instead, or lifted by a power of two, they cost as much, and lifted they put outputs off by 1.1 times as much.)
__device__ __forceinline__ f32x2 pow2_pair(f32x2 v, float c, float c_rest, float least) {
  constexpr float LN2 = 0.693147180559945f;
  float x, y;
  unpack2(v, x, y);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(least));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(y) : "f"(least));
  const f32x2 z = pack2(x, y), t = mul2(z, both(c)), over = fma2(z, both(-c_rest), fma2(z, both(-c), t));
  unpack2(t, x, y);
  asm("ex2.approx.f32 %0, %0;" : "+f"(x));
  asm("ex2.approx.f32 %0, %0;" : "+f"(y));
  const f32x2 r = pack2(x, y);
  return fma2(mul2(r, both(-LN2)), over, r);
}
__device__ __forceinline__ f32x2 exp_pair(f32x2 x) { return pow2_pair(x, 1.44269502162933349609f, 1.92596299e-8f, -150.f); }

// The warp's number in its group of four, known to be the same in all lanes (addresses in TMEM are the warp's)
__device__ __forceinline__ int group_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5) & 3, 0); }
// by one thread
__device__ __forceinline__ void init_hand_overs(AttnTail& sm) {
  sm.dead = 0;
  mbar_init(smem_u32(&sm.q_full), 8);
  for (int i = 0; i < 2; ++i) {
    mbar_init(smem_u32(&sm.s_full[i]), 1);
    mbar_init(smem_u32(&sm.p_full[i]), 8);
    for (int w = 0; w < 4; ++w) mbar_init(smem_u32(&sm.m_full[i][w]), 1);
  }
  mbar_init(smem_u32(&sm.o_full), 1);
  mbar_init(smem_u32(&sm.drain), 1);
}
// by all threads; ends with TMEM allocated and the barriers seen by all
__device__ __forceinline__ uint32_t take_tmem(AttnTail& sm, int warp) {
  if (warp == ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  return __shfl_sync(0xffffffffu, sm.tmem, 0);                     // (known to be the same in all lanes: instructions take it as it is)
}
__device__ __forceinline__ void give_tmem_back(uint32_t tmem, int warp) {
  tcgen05_fence_before();
  __syncthreads();
  if (warp == ISSUER) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
// by all threads, at the end: products and loads in flight (loads(): by one thread) end before shared memory and TMEM are given back
template <class Loads> __device__ __forceinline__ void leave(AttnTail& sm, uint32_t tmem, int warp, int* timeouts, const Loads& loads) {
  volatile int* dead = &sm.dead;
  if (__syncthreads_or(*dead)) {
    if (threadIdx.x == 0) atomicAdd_system(timeouts, 1);
    if (warp == ISSUER) {
      commit_if(elect_one(), smem_u32(&sm.drain));
      wait_in_flight(smem_u32(&sm.drain), 0u);
      if ((threadIdx.x & 31) == 0) loads();
    }
  }
  give_tmem_back(tmem, warp);
}

// A block's weights, one part of them, times one part of its values; `vb`: the descriptor of [KEYS][128 columns] in two slabs
template <int KEYS> __device__ __forceinline__ void issue_values(uint32_t one, uint32_t tmem, int s, int part, uint64_t vb, bool first) {
  constexpr uint32_t idesc = make_idesc(ROWS, D) | (1u << 16);     // the values lie with the keys as rows
#pragma unroll
  for (int k = 0; k < KEYS / 16; ++k) mma_tmem_a_if(one, tmem + SUMS, tmem + s * GROUP + WEIGHTS + part * (KEYS / 2) + k * 8, vb + k * 128, idesc, !first || k > 0);
}

// What a block's weights take from the block before: hands its maximum `top` of a thread's row to the other group's warp of the same rows and returns the one before it (false: a wait ran out)
__device__ __forceinline__ bool hand_over_top(AttnTail& sm, int s, int it, float& top, float& before) {
  const int w = group_warp(), lane = threadIdx.x & 31, r = w * 32 + lane;
  before = -INFINITY;
  if (it > 0) {
    if (!warp_wait(smem_u32(&sm.m_full[s ^ 1][w]), ((it - 1) >> 1) & 1, &sm.dead)) return false;
    before = sm.top[s ^ 1][r];
  }
  top = fmaxf(top, before);
  sm.top[s][r] = top;
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&sm.m_full[s][w]));
  return true;
}
// Two weights as packed pairs of their three parts (split3_finite, mma.cuh)
__device__ __forceinline__ void split_pair(f32x2 w, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  float x, y;
  unpack2(w, x, y);
  hi = pack_bf16x2(x, y);
  unpack_bf16x2(hi, x, y);
  const f32x2 rest = fma2(pack2(x, y), both(-1.f), w);
  unpack2(rest, x, y);
  mid = pack_bf16x2(x, y);
  unpack_bf16x2(mid, x, y);
  unpack2(fma2(pack2(x, y), both(-1.f), rest), x, y);
  lo = pack_bf16x2(x, y);
}

// The sums of all blocks of a thread's row; false: a wait ran out.  (The weights' sum in 64 bits: its error is that of every column.)
__device__ __forceinline__ bool sum_blocks(AttnTail& sm, uint32_t tmem, int n, f32x2 (&O)[D / 2], double& l) {
  volatile int* dead = &sm.dead;
  const int w = group_warp(), lane = threadIdx.x & 31, r = w * 32 + lane;
  const uint32_t to = tmem + SUMS + ((uint32_t)(w * 32) << 16);
  bool alive = true;
  l = 0.0;
#pragma unroll
  for (int c = 0; c < D / 2; ++c) O[c] = 0ull;
  if (lane == 0) mbar_arrive(smem_u32(&sm.p_full[0]));             // nothing is in the first block's place
#pragma unroll 1
  for (int it = 0; it < n; ++it) {
    if (!(alive = warp_wait(smem_u32(&sm.o_full), it & 1, dead))) break;
    tcgen05_fence_after();
    const float2 add = sm.add[it & 3][r];
    l = fma(l, (double)add.x, (double)add.y);
#pragma unroll
    for (int c = 0; c < D; c += 32) {
      uint32_t v[32];
      tmem_ld32(to + c, v);
      tmem_ld_wait();
      if (c == D - 32) {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.p_full[(it + 1) & 1]));
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) O[c / 2 + i] = fma2(O[c / 2 + i], both(add.x), pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
    }
  }
  return alive;
}

// A warp's 32 rows by way of 16 KB of shared memory at `place`, times `inv` of their threads: put(i, y) for row i and columns 4 lane .. 4 lane + 3, for neighbouring lanes to write neighbouring
// columns; before that gate(i, y) if `gated`, four rows at a time (one: 2 us more a tile, two 0.9, eight as four).  Returns the rows among the first `rows` whose sums are not finite, which are not put: they are for the caller to form again.  With sums of a wait that ran
// out (`alive` false; `inv` is NaN) there are none, and every row is put.  (Little code, and what is not needed in one piece to skip: it is run once, and instructions come slowly then.)
template <class Gate, class Put>
__device__ __forceinline__ unsigned rows_out(uint8_t* place, const f32x2 (&O)[D / 2], float inv, bool alive, int rows, bool gated, const Gate& gate, const Put& put) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < D; c += 4) {
    float4 y;
    unpack2(O[c / 2], y.x, y.y);
    unpack2(O[c / 2 + 1], y.z, y.w);
    reinterpret_cast<float4*>(place)[lane * (D / 4) + ((c / 4) ^ (lane & 7))] = y;
  }
  f32x2 probe[4] = {0ull, 0ull, 0ull, 0ull};                       // NaN if a sum is not finite
#pragma unroll
  for (int c = 0; c < D / 2; ++c) probe[c & 3] = fma2(O[c], 0ull, probe[c & 3]);
  float p0, p1;
  unpack2(add2(add2(probe[0], probe[1]), add2(probe[2], probe[3])), p0, p1);
  const unsigned again = __ballot_sync(0xffffffffu, alive && lane < rows && p0 + p1 != 0.f);
  cp_async_wait<0>();                                              // (gates)
  __syncwarp();
  auto row = [&](int i) {
    const float4 y = reinterpret_cast<const float4*>(place)[i * (D / 4) + (lane ^ (i & 7))];
    const float f = __shfl_sync(0xffffffffu, inv, i);
    return make_float4(y.x * f, y.y * f, y.z * f, y.w * f);
  };
  auto out = [&](auto together, auto with) {
    constexpr int N = decltype(together)::value;
#pragma unroll 1
    for (int i0 = 0; i0 < 32 && i0 < rows; i0 += N) {
      float4 y[N];
#pragma unroll
      for (int i = 0; i < N; ++i) y[i] = row(i0 + i);
#pragma unroll
      for (int i = 0; i < N; ++i) with(i0 + i, y[i]);
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (i0 + i < rows && !((again >> (i0 + i)) & 1u)) put(i0 + i, y[i]);
    }
  };
  if (gated) out(std::integral_constant<int, 4>(), gate);
  else out(std::integral_constant<int, 8>(), [](int, float4&) {});
  return again;
}

template <class Kernel> bool registers_suffice(Kernel* kernel) {   // those that the warps trade must be those that the block gets
  cudaFuncAttributes at{};
  return cudaFuncGetAttributes(&at, kernel) == cudaSuccess && at.numRegs * THREADS >= 128 * (2 * SOFTMAX_REGS + SUM_REGS + OTHER_REGS);
}

}  // namespace
