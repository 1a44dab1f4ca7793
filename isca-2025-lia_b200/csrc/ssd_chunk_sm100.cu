// The state-space recurrence of linear_scan.cu (S = g S + dt B x^T, o = S^T C + D x; 128 state rows, heads of 64 k columns) over long portions: chunks of 128 tokens, all
// chunks at once, as tcgen05 contractions.
//
// With P[t][s] the product of the decays after s up to t and S the state before the chunk:
//     o = (P o C B^T) (dt x) + P[t][-1] (C S)  + D x           S' = P[last][-1] S + B^T (w x),  w[s] = P[last][s] dt[s]
// Token by token a head's state costs three FMAs per element and token on the CUDA cores, and a token waits for the one before it.  Here only S' is a chain:
//   states   every chunk's B^T (w x), 128 x 64 per head                              -> workspace
//   carry    the states before every chunk, element by element, and the last one     -> workspace, in place
//   outputs  C B^T once per group of heads, then per head the two products with C and with the weights
// A CTA takes a chunk and some heads of one group, whose B and C it splits once.  All operands are fp32 numbers and enter as three fp16 parts each, all products but lo lo, whose accumulators
// gather them by size (hi hi | hi mid, mid hi, mid mid | the rest); the parts of one operand lie side by side, so that an instruction can take several.
// The tensor cores cut their sums off below the 24th bit, eight instructions in a row off by 1.8e-7.  So each row of A and column of B is brought, by a power of two, to numbers below 2^15, and
// its hi parts are whole multiples, of at most 256, of 2^7: 128 products of two such numbers have a sum below 2^23 of their unit, which the accumulator holds exactly.  The rest of a number
// goes on in two parts of 11 bits and a sign, the second times 2^11 against fp16's smallest numbers: nothing of fp32 is lost down to 2^-26 of the row's or column's largest number
// (and 2^-51 of that at most below), so that a token is as exact beside a large one as alone.  (Two bf16 parts for the rest kept 16 to 18 bits of a number below 2^-8 of the largest: 1e3 times the others in the last token of a
// chunk put the tokens before it off by 1.2e-6.)  There the sums of the second accumulator are the result, and smaller products go into it first: what is cut off each of them is then
// off a smaller sum.
// The weights P o C B^T go from registers to TMEM and are the A operand from there.
//
// 2048 tokens, 64 heads of 64 in 8 groups: 270 us token by token -> 48 states + 10 carry + 88 outputs (with bf16 parts, and D x from them, 49 + 10 + 73); Mamba's mixer 405 -> 278 (270).  Against 64 bits, same inputs: outputs off by 5.9e-8 (token loop
// 6.6e-8), states by 0.95e-8 (1.5e-8); decays near 1: 4.6e-8 (11.1e-8) and 4.5e-8 (39.8e-8).
//
// The weights are products of decays (never quotients or differences of logarithms).  Inputs that are not finite, or so large that a chunk's sums could overflow where the token loop's
// would not, are left to the token loop, head by head (`flags`): there a bad value reaches the tokens after it and no other.
//
// Every wait is bounded: a CTA of `states` that gave up hands its heads to the token loop, one of `outputs` leaves NaN and counts itself (lia_moe_timeouts_seen).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "mma.cuh"
#include "umma.cuh"

int* lia_timeout_word();                                           // moe_sm100.cu
int ssd_scan_tokens(const float* B, const float* C, const float* x, int ld, const float* gates, const float* D, float* St, const int* segs, int tok0, int span, int below, int longs,
                    const int* flags, const float* after, bool single, int nseg, int H, int G, int N, int vdim, float* o, cudaStream_t stream);      // linear_scan.cu

namespace {

constexpr int L = 128, N = 128, P = 64;        // tokens of a chunk, rows of the state, columns of a unit (a head, or 64 columns of one)
constexpr int MAX_UNITS = 8;                   // per CTA
// Portions of fewer tokens go token by token.  One portion of 256 | 384 | 448 | 512 | 2048 tokens, 64 heads: 37 | 54 | 62 | 70 | 269 us there and 47 | 55 | 55 | 57 | 152 here; 16 heads: 37 | 54 |
// 62 | 70 | 266 and 42 | 43 | 45 | 47 | 65; 64 heads beside 32 single tokens: 56 | 82 | 95 | 108 and 78 | 90 | 92 | 95.  (Where the chunks of several portions are little more than the SMs a longer one
// can still lose: four of 640, 32 heads, 134 and 159.)
constexpr int SHORT = 448;
constexpr int TILE = 2 * L * 128;              // one part of B or C: two slabs of 64 rows of the state, 128 bytes a token
constexpr int UNIT = L * 128;                  // one part of a unit's x, or of half its state
constexpr float BIG = 1073741824.f, BIG_STATE = 1.2e30f;           // 2^30, 2^100

struct SsdArgs {
  const float *B, *C, *x;
  int ld;
  const float *gates, *D;
  float* St;
  const int* segs;
  int nseg, H, G, U, per_head;                 // U: units in all; per_head: units of a head
  float* o;
  float *states, *after;                       // [slots][U][P][N]; [longs][U][P][N]: after the tokens of the portions of SHORT tokens and more, in order
  float2* totals;                              // [slots][U]: the product of a chunk's decays, and what is left of it
  int *bad, *flags;                            // [slots][U], [longs][H]
  int slots, longs;
  int tok0, span, split, per_cta;              // the tokens tok0 .. tok0 + span - 1 of every portion; a group's units in `split` CTAs of `per_cta`
  int* timeouts;
};

__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The products of two operands in three parts each: part of A (bits 0-1), first part of B (2-3) and how many of its parts (4-5), which accumulator (6-7), whether it begins that (8).
// (The instructions are issued from loops: unrolled they would not fit into the instruction cache beside the other warps' code.)
constexpr int product_code(int a, int b, int parts, int to, int first) { return a | b << 2 | parts << 4 | to << 6 | first << 8; }
__constant__ int PRODUCTS[7] = {product_code(2, 0, 1, 2, 1), product_code(2, 1, 1, 2, 0), product_code(1, 2, 1, 2, 0), product_code(1, 1, 1, 1, 1), product_code(1, 0, 1, 1, 0),
                                product_code(0, 0, 1, 0, 1), product_code(0, 1, 2, 1, 0)};
__constant__ int SINGLES[8] = {product_code(2, 0, 1, 2, 1), product_code(2, 1, 1, 2, 0), product_code(1, 2, 1, 2, 0), product_code(0, 2, 1, 2, 0),
                               product_code(1, 1, 1, 1, 1), product_code(1, 0, 1, 1, 0), product_code(0, 1, 1, 1, 0), product_code(0, 0, 1, 0, 1)};
constexpr float LOW = 1.f / 2048.f;            // what the third accumulator counts for
__device__ __forceinline__ float gathered(uint32_t a, uint32_t b, uint32_t c) { return __uint_as_float(a) + fmaf(__uint_as_float(c), LOW, __uint_as_float(b)); }
// K = 128.  Steps in 16-byte units: a part, 64 of the contracted numbers, 16 of them (A in TMEM: in columns, as is `a`); `width`: columns of one part of B, and of an accumulator.
struct Operand {
  uint64_t at;
  uint32_t part, slab, step;
};
template <bool tmem_a> __device__ __forceinline__ void issue(uint32_t one, const int* codes, int count, uint32_t d, const Operand& A, const Operand& B, int width, uint32_t major) {
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    const int code = codes[i];
    constexpr uint32_t bf16_operands = 1u << 7 | 1u << 10;           // fp16: neither bit
    const uint32_t idesc = (make_idesc(128, 0) & ~bf16_operands) | major | (uint32_t)(((code >> 4 & 3) * width) >> 3) << 17, to = d + (code >> 6 & 3) * width;
    uint64_t a = A.at + (code & 3) * A.part, b = B.at + (code >> 2 & 3) * B.part;
    uint32_t accumulate = !(code >> 8 & 1);
#pragma unroll 1
    for (int half = 0; half < 2; ++half, a += A.slab, b += B.slab) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (tmem_a) mma_tmem_a_if(one, to, (uint32_t)a + k * A.step, b + k * B.step, idesc, accumulate);
        else mma_if(one, to, a + k * A.step, b + k * B.step, idesc, accumulate);
        accumulate = 1u;
      }
    }
  }
}

struct Chunk {
  int seg, slot, row0, tokens;                 // tokens < L at a portion's end
  bool first;
};
__device__ __forceinline__ int window_tokens(const SsdArgs& p, int k) {
  const int len = p.segs[4 * k + 3];
  return len >= SHORT ? min(max(len - p.tok0, 0), p.span) : 0;
}
// the i-th chunk of the step (a whole warp asks)
__device__ __forceinline__ bool locate(const SsdArgs& p, int i, Chunk& c) {
  const int lane = threadIdx.x & 31;
  for (int k0 = 0; k0 < p.nseg; k0 += 32) {
    const int k = k0 + lane, tokens = k < p.nseg ? window_tokens(p, k) : 0, n = (tokens + L - 1) / L;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    const unsigned past = __ballot_sync(0xffffffffu, sum > i);
    if (past) {
      const int at = __ffs(past) - 1, chunk = i - __shfl_sync(0xffffffffu, sum - n, at);
      c.seg = k0 + at;
      c.slot = p.segs[4 * c.seg];
      c.row0 = p.segs[4 * c.seg + 2] + p.tok0 + chunk * L;
      c.tokens = min(L, __shfl_sync(0xffffffffu, tokens, at) - chunk * L);
      c.first = chunk == 0;
      return true;
    }
    i -= __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}

// The rank-th portion of SHORT tokens and more, and the chunks before it (a whole warp asks)
__device__ __forceinline__ bool nth_long(const SsdArgs& p, int rank, int& seg, int& before) {
  const int lane = threadIdx.x & 31;
  before = 0;
  for (int k0 = 0; k0 < p.nseg; k0 += 32) {
    const int k = k0 + lane;
    const unsigned taken = __ballot_sync(0xffffffffu, k < p.nseg && p.segs[4 * k + 3] >= SHORT);
    const int found = __popc(taken), at = rank < found ? (int)__fns(taken, 0, rank + 1) : 32;
    int n = k < p.nseg && lane < at ? (window_tokens(p, k) + L - 1) / L : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    before += n;
    if (rank < found) {
      seg = k0 + at;
      return true;
    }
    rank -= found;
  }
  return false;
}

__device__ __forceinline__ void load8(const float* src, bool live, float* v) {
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
  if (live) {
    a = *reinterpret_cast<const float4*>(src);
    b = *reinterpret_cast<const float4*>(src + 4);
  }
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
// The power of two that brings numbers up to `most` below 2^15 (those of a row of less than 2^-100 stay smaller), and its inverse
__device__ __forceinline__ float scale_of(float most) { return __uint_as_float((268u << 23) - max(__float_as_uint(most) & 0x7f800000u, 27u << 23)); }
__device__ __forceinline__ float inverse_of(float scale) { return __uint_as_float((254u << 23) - __float_as_uint(scale)); }
__device__ __forceinline__ uint32_t pack_half2(float x, float y) {
  const __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void split3(float x, float y, float sx, float sy, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  constexpr float R = 1610612736.f;            // its last bit is 2^7: added and taken away again it rounds to a multiple of that
  x *= sx, y *= sy;
  const float hx = __fsub_rn(__fadd_rn(x, R), R), hy = __fsub_rn(__fadd_rn(y, R), R), dx = x - hx, dy = y - hy;          // exact differences
  hi = pack_half2(hx, hy);
  mid = pack_half2(dx, dy);
  const float2 m = __half22float2(*reinterpret_cast<const __half2*>(&mid));
  lo = pack_half2((dx - m.x) * 2048.f, (dy - m.y) * 2048.f);
}
// 8 neighbouring numbers as 16 bytes in each of three tiles `stride` bytes apart, with a scale each (or one: each = 0)
template <int each> __device__ __forceinline__ void put_parts(uint32_t addr, uint32_t stride, const float* v, const float* s) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split3(v[2 * i], v[2 * i + 1], s[each * 2 * i], s[each * (2 * i + 1)], h[i], m[i], l[i]);
  st_shared16(addr, h[0], h[1], h[2], h[3]);
  st_shared16(addr + stride, m[0], m[1], m[2], m[3]);
  st_shared16(addr + 2 * stride, l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ float most8(const float* v) {
  return fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))), fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fabsf(v[7]))));
}
// The scales of 8 neighbouring columns from `rows` rows of maxima
template <int rows, int cols> __device__ __forceinline__ void scales_of(const float (&m)[rows][cols], int col, float* r) {
#pragma unroll
  for (int e = 0; e < 8; e += 4) {
    float4 a = *reinterpret_cast<const float4*>(&m[0][col + e]);
#pragma unroll
    for (int k = 1; k < rows; ++k) {
      const float4 b = *reinterpret_cast<const float4*>(&m[k][col + e]);
      a = make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
    }
    r[e] = scale_of(a.x), r[e + 1] = scale_of(a.y), r[e + 2] = scale_of(a.z), r[e + 3] = scale_of(a.w);
  }
}
// A row of 128 numbers over 16 lanes, 8 each: the largest
__device__ __forceinline__ float most_of_row(const float* v) {
  float m = most8(v);
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// A warp's view of a unit's decays over a chunk; a lane has the tokens 4 lane .. 4 lane + 3.  Products in 64 bits, rounded once where they are used: rounded one by one they are off by the
// same factor for a whole state, which no sum averages out (2.1e-7 of the outputs at decays near 1, token by token 1.05e-7).
struct Decays {
  float a[4], dt[4];
  double upto[4], after[4], block[4];          // of the token's block of 32: up to it, after it; of the chunk's four blocks
};
__device__ __forceinline__ Decays decays_of(const SsdArgs& p, const Chunk& c, int h) {
  const int lane = threadIdx.x & 31;
  Decays d;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = 4 * lane + i;
    const float* gp = p.gates + (size_t)(c.row0 + t) * 2 * p.H + h;
    d.dt[i] = t < c.tokens ? gp[0] : 0.f;
    d.a[i] = t < c.tokens ? gp[p.H] : 1.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) d.upto[i] = i ? d.upto[i - 1] * d.a[i] : (double)d.a[0];
  d.after[3] = 1.0;
#pragma unroll
  for (int i = 2; i >= 0; --i) d.after[i] = d.after[i + 1] * d.a[i + 1];
  double up = d.upto[3], down = up;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, up, o), n = __shfl_down_sync(0xffffffffu, down, o);
    if ((lane & 7) >= o) up *= u;
    if ((lane & 7) + o < 8) down *= n;
  }
  const double lead = __shfl_up_sync(0xffffffffu, up, 1), tail = __shfl_down_sync(0xffffffffu, down, 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (lane & 7) d.upto[i] *= lead;
    if ((lane & 7) != 7) d.after[i] *= tail;
    d.block[i] = __shfl_sync(0xffffffffu, up, 8 * i + 7);
  }
  return d;
}

// ------------------------------------------------------------------------------------------------ states
// 416 threads: warps 0-3 drain one of two accumulators (lane = row of the state), warps 4-11 split x (two buffers), warp 12 issues.
// TMEM: 2 x 192 columns.
constexpr int ST_THREADS = 416;
struct StBars {
  uint64_t x_full[2], x_empty[2], scaled[2], acc_full[2], acc_empty[2], drain;             // scaled: the scales that a unit was split by are written
};
struct StSmem {
  alignas(16) float w[MAX_UNITS][L];
  alignas(16) float most_b[8][N], most_x[8][P];                    // by warp
  alignas(16) float inv_x[MAX_UNITS][P];                           // the scales' inverses
  float inv_b[N];
  float total[MAX_UNITS], total_rest[MAX_UNITS];
  int bad[MAX_UNITS], bad_all, dead;
  uint32_t tmem;
  StBars bars;
};
constexpr int ST_BYTES = 3 * TILE + 2 * 3 * UNIT + sizeof(StSmem) + 1024;

__global__ void __launch_bounds__(ST_THREADS, 1) ssd_states_kernel(const SsdArgs p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u, xs = base + 3 * TILE;
  StSmem& sm = *reinterpret_cast<StSmem*>(raw + (base - smem_u32(raw)) + 3 * TILE + 6 * UNIT);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* dead = &sm.dead;
  if (tid == 0) {
    sm.dead = sm.bad_all = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sm.bars.x_full[i]), 8);
      mbar_init(smem_u32(&sm.bars.x_empty[i]), 1);
      mbar_init(smem_u32(&sm.bars.scaled[i]), 1);
      mbar_init(smem_u32(&sm.bars.acc_full[i]), 1);
      mbar_init(smem_u32(&sm.bars.acc_empty[i]), 4);
    }
    mbar_init(smem_u32(&sm.bars.drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < MAX_UNITS) sm.bad[tid] = 0;
  pdl_wait();
  Chunk c;
  const int per_group = p.U / p.G, group = blockIdx.y / p.split, u0 = group * per_group + (blockIdx.y % p.split) * p.per_cta;
  const int units = min(p.per_cta, (group + 1) * per_group - u0);
  if (units <= 0 || !locate(p, blockIdx.x, c)) return;             // the same for all threads
  if (warp == 12) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();                                                 // bad[] is clear

  // what a token's x counts for in the state after the chunk
  for (int j = warp; warp < 4 && j < units; j += 4) {
    const Decays d = decays_of(p, c, (u0 + j) / p.per_head);
    bool fine = true;
    double later = 1.0, all = 1.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      fine = fine && d.a[i] >= 0.f && d.a[i] <= 1.f && fabsf(d.dt[i]) < BIG;
      if (i > (lane >> 3)) later *= d.block[i];
      all *= d.block[i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) sm.w[j][4 * lane + i] = (float)(d.dt[i] * (d.after[i] * later));
    if (lane == 0) {
      sm.total[j] = (float)all;
      sm.total_rest[j] = (float)(all - (double)(float)all);
    }
    if (!__all_sync(0xffffffffu, fine) && lane == 0) sm.bad[j] = 1;
  }
  if (warp >= 4 && warp < 12) {                                    // B: a thread has 8 tokens of 8 rows of the state; a scale per row of the state
    const int th = tid - 128, piece = th & 15;
    float v[8][8], most[8] = {};
    bool fine = true;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = (th >> 4) + i * 16;
      load8(p.B + (size_t)(c.row0 + t) * p.ld + group * N + piece * 8, t < c.tokens, v[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        fine = fine && fabsf(v[i][e]) < BIG;
        most[e] = fmaxf(most[e], fabsf(v[i][e]));
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) most[e] = fmaxf(most[e], __shfl_xor_sync(0xffffffffu, most[e], 16));
    if (lane < 16) {
#pragma unroll
      for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(&sm.most_b[warp - 4][piece * 8 + e]) = make_float4(most[e], most[e + 1], most[e + 2], most[e + 3]);
    }
    if (!fine) sm.bad_all = 1;
    asm volatile("bar.sync 2, 256;" ::: "memory");
    scales_of(sm.most_b, piece * 8, most);
    if (th < 16) {
#pragma unroll
      for (int e = 0; e < 8; ++e) sm.inv_b[piece * 8 + e] = inverse_of(most[e]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = (th >> 4) + i * 16;
      put_parts<1>(base + (piece >> 3) * (TILE / 2) + t * 128 + (((piece & 7) ^ (t & 7)) << 4), TILE, v[i], most);
    }
    fence_proxy_async_smem();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem, 0);

  const uint32_t one = elect_one();
  if (warp == 12) {
    constexpr uint32_t mn = (1u << 15) | (1u << 16);               // both operands lie with the contracted tokens as rows
#pragma unroll 1
    for (int j = 0; j < units; ++j) {
      const int b = j & 1;
      const uint32_t parity = (j >> 1) & 1;
      if (!warp_wait(smem_u32(&sm.bars.x_full[b]), parity, dead) || !warp_wait(smem_u32(&sm.bars.acc_empty[b]), parity ^ 1u, dead)) break;
      if (one) mbar_arrive(smem_u32(&sm.bars.scaled[b]));
      tcgen05_fence_after();
      const uint32_t d = tmem + b * 192, xb = xs + b * 3 * UNIT;
      issue<false>(one, PRODUCTS, 7, d, Operand{make_smem_desc_mn(base, TILE / 2), TILE >> 4, 512, 128}, Operand{make_smem_desc_mn(xb, UNIT), UNIT >> 4, 512, 128}, 64, mn);
      commit_if(one, smem_u32(&sm.bars.x_empty[b]));
      commit_if(one, smem_u32(&sm.bars.acc_full[b]));
    }
  } else if (warp >= 4) {
    const int th = tid - 128;
    bool alive = true;
    float next[4][8];
    auto get = [&](int j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = th + i * 256, t = e >> 3;
        load8(p.x + (size_t)(c.row0 + t) * p.ld + (u0 + j) * P + (e & 7) * 8, t < c.tokens, next[i]);
      }
    };
    get(0);
    for (int j = 0; j < units; ++j) {
      const int b = j & 1;
      float v[4][8];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i >> 3][i & 7] = next[i >> 3][i & 7];
      if (j + 1 < units) get(j + 1);
      bool fine = true;
      float most[8] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float w = sm.w[j][(th + i * 256) >> 3];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          fine = fine && fabsf(v[i][k]) < BIG;
          v[i][k] *= w;
          most[k] = fmaxf(most[k], fabsf(v[i][k]));
        }
      }
      if (!fine) sm.bad[j] = 1;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        most[k] = fmaxf(most[k], __shfl_xor_sync(0xffffffffu, most[k], 8));
        most[k] = fmaxf(most[k], __shfl_xor_sync(0xffffffffu, most[k], 16));
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");               // the last unit's are read
      if (lane < 8) {
#pragma unroll
        for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(&sm.most_x[warp - 4][lane * 8 + e]) = make_float4(most[e], most[e + 1], most[e + 2], most[e + 3]);
      }
      asm volatile("bar.sync 2, 256;" ::: "memory");
      scales_of(sm.most_x, (lane & 7) * 8, most);
      if (th < 8) {
#pragma unroll
        for (int e = 0; e < 8; ++e) sm.inv_x[j][th * 8 + e] = inverse_of(most[e]);
      }
      if (alive) alive = warp_wait(smem_u32(&sm.bars.x_empty[b]), ((j >> 1) & 1) ^ 1u, dead);
      if (!alive) continue;                                        // (the others still meet at the barriers)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = th + i * 256, t = e >> 3, piece = e & 7;
        put_parts<1>(xs + b * 3 * UNIT + t * 128 + ((piece ^ (t & 7)) << 4), UNIT, v[i], most);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.bars.x_full[b]));
    }
  } else {
    // a bad value could also hide in C
    bool fine = true;
    const float* cp = p.C + (size_t)c.row0 * p.ld + group * N;
#pragma unroll 8
    for (int e = tid; e < c.tokens * 32; e += 128) {
      const float4 v = *reinterpret_cast<const float4*>(cp + (size_t)(e >> 5) * p.ld + (e & 31) * 4);
      fine = fine && fabsf(v.x) < BIG && fabsf(v.y) < BIG && fabsf(v.z) < BIG && fabsf(v.w) < BIG;
    }
    if (!fine) sm.bad_all = 1;
    for (int j = 0; j < units; ++j) {
      const int b = j & 1;
      if (!warp_wait(smem_u32(&sm.bars.scaled[b]), (j >> 1) & 1, dead) || !warp_wait(smem_u32(&sm.bars.acc_full[b]), (j >> 1) & 1, dead)) break;
      tcgen05_fence_after();
      const float inv = sm.inv_b[warp * 32 + lane];
      float* dst = p.states + ((size_t)blockIdx.x * p.U + u0 + j) * P * N + warp * 32 + lane;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[3][32];
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_ld32(tmem + b * 192 + i * 64 + half * 32 + ((uint32_t)(warp * 32) << 16), v[i]);
        tmem_ld_wait();
        if (half == 1) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sm.bars.acc_empty[b]));
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) dst[(half * 32 + i) * N] = gathered(v[0][i], v[1][i], v[2][i]) * inv * sm.inv_x[j][half * 32 + i];
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (tid < units) {
    p.bad[(size_t)blockIdx.x * p.U + u0 + tid] = sm.bad[tid] | sm.bad_all | *dead;
    p.totals[(size_t)blockIdx.x * p.U + u0 + tid] = make_float2(sm.total[tid], sm.total_rest[tid]);
  }
  if (*dead) {
    if (warp == 12) {                                              // products in flight end before shared memory and TMEM are given back
      commit_if(one, smem_u32(&sm.bars.drain));
      wait_in_flight(smem_u32(&sm.bars.drain), 0u);
    }
    __syncthreads();
  }
  if (warp == 12) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------ carry
constexpr int CARRY = 256;
// a thread carries four elements of a unit's state over its portion's chunks; 8 blocks per unit
__global__ void __launch_bounds__(CARRY, 4) ssd_carry_kernel(const SsdArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  const int u = blockIdx.x >> 3, rank = blockIdx.y;
  int seg, before;
  if (!nth_long(p, rank, seg, before)) return;
  const int n = (window_tokens(p, seg) + L - 1) / L;
  if (n == 0 || before + n > p.slots) return;
  const int head0 = u / p.per_head * p.per_head;
  int bad = 0;
  for (int e = threadIdx.x; e < n * p.per_head; e += CARRY) bad |= p.bad[(size_t)(before + e / p.per_head) * p.U + head0 + e % p.per_head];
  const float4* start = reinterpret_cast<const float4*>(p.St) + ((size_t)p.segs[4 * seg] * p.U + head0) * (P * N / 4);      // what the head starts from, all of it
  for (int k = 0; k < p.per_head; ++k) {
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = start[(size_t)k * (P * N / 4) + i * CARRY + threadIdx.x];
#pragma unroll
    for (int i = 0; i < 8; ++i) bad |= !(fabsf(v[i].x) < BIG_STATE && fabsf(v[i].y) < BIG_STATE && fabsf(v[i].z) < BIG_STATE && fabsf(v[i].w) < BIG_STATE);
  }
  bad = __syncthreads_or(bad);
  if ((blockIdx.x & 7) == 0 && threadIdx.x == 0) p.flags[(size_t)rank * p.H + u / p.per_head] = bad;
  const size_t at = (size_t)u * (P * N / 4) + (blockIdx.x & 7) * CARRY + threadIdx.x, step = (size_t)p.U * (P * N / 4);
  float4* st = reinterpret_cast<float4*>(p.states) + (size_t)before * step + at;
  const float2* total = p.totals + (size_t)before * p.U + u;
  float4 S = reinterpret_cast<const float4*>(p.St)[(size_t)p.segs[4 * seg] * step + at];
  for (int c0 = 0; c0 < n; c0 += 4) {
    float4 local[4];
    float2 f[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (c0 + i < n) {
        local[i] = st[(size_t)(c0 + i) * step];
        f[i] = total[(size_t)(c0 + i) * p.U];
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (c0 + i < n) {
        st[(size_t)(c0 + i) * step] = S;
        S.x = fmaf(f[i].x, S.x, fmaf(f[i].y, S.x, local[i].x));
        S.y = fmaf(f[i].x, S.y, fmaf(f[i].y, S.y, local[i].y));
        S.z = fmaf(f[i].x, S.z, fmaf(f[i].y, S.z, local[i].z));
        S.w = fmaf(f[i].x, S.w, fmaf(f[i].y, S.w, local[i].w));
      }
  }
  reinterpret_cast<float4*>(p.after)[(size_t)rank * step + at] = S;     // (the token loop may still need what is in St)
}

// ------------------------------------------------------------------------------------------------ outputs
// 512 threads.  Warps 0-7 but 4 make the weights (lane = token t; warps 0-3 the first 64 tokens s, 5-7 the others) from C B^T, warp 4, whose weights are all zero, issues,
// warps 8-11 put the outputs together, warps 12-15 split the units' states and x.  Shared memory: C | B, whose place the states and x take.
// TMEM: weights 192 columns, accumulators 192, C B^T 128 (its parts before: 384).
constexpr int OUT_THREADS = 512;
struct OutBars {
  uint64_t cb_full, cb_read, s_full, x_full, w_full, inter_scaled, inter_full, inter_read, intra_scaled, intra_full, intra_read, drain;     // scaled: as above
};
struct OutSmem {
  alignas(16) float dt[MAX_UNITS][L], a[MAX_UNITS][L], pre[MAX_UNITS][L];     // pre: the decays from the chunk's start up to a token
  alignas(16) float upto[MAX_UNITS][L], after[MAX_UNITS][L], block[MAX_UNITS][4];          // within its block of 32: up to it; after it, times its dt; the blocks' own
  alignas(16) float most_x[4][P];
  float most_w[2][L];
  alignas(16) float inv_b[L], inv_c[L], inv_w[2][L], inv_s[2][P], inv_x[P];                // the scales' inverses; [2]: one unit's while the last one's are read
  int dead;
  uint32_t tmem;
  OutBars bars;
};
constexpr int OUT_BYTES = 6 * TILE + sizeof(OutSmem) + 1024;
constexpr int S_HALF = 3 * P * 128;            // the states' slab of 64 rows of the state: [hi | mid | lo][64 columns][128 bytes]

__global__ void __launch_bounds__(OUT_THREADS, 1) ssd_outputs_kernel(const SsdArgs p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u, second = base + 3 * TILE, ss = second, xs = second + 2 * S_HALF;
  OutSmem& sm = *reinterpret_cast<OutSmem*>(raw + (base - smem_u32(raw)) + 6 * TILE);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* dead = &sm.dead;
  if (tid == 0) {
    sm.dead = 0;
    mbar_init(smem_u32(&sm.bars.cb_full), 1);
    mbar_init(smem_u32(&sm.bars.cb_read), 8);
    mbar_init(smem_u32(&sm.bars.s_full), 4);
    mbar_init(smem_u32(&sm.bars.x_full), 4);
    mbar_init(smem_u32(&sm.bars.w_full), 7);
    mbar_init(smem_u32(&sm.bars.inter_scaled), 1);
    mbar_init(smem_u32(&sm.bars.intra_scaled), 1);
    mbar_init(smem_u32(&sm.bars.inter_full), 1);
    mbar_init(smem_u32(&sm.bars.inter_read), 4);
    mbar_init(smem_u32(&sm.bars.intra_full), 1);
    mbar_init(smem_u32(&sm.bars.intra_read), 4);
    mbar_init(smem_u32(&sm.bars.drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  Chunk c;
  const int per_group = p.U / p.G, group = blockIdx.y / p.split, u0 = group * per_group + (blockIdx.y % p.split) * p.per_cta;
  const int units = min(p.per_cta, (group + 1) * per_group - u0);
  if (units <= 0 || !locate(p, blockIdx.x, c)) return;             // the same for all threads
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  {                                                                // C by warps 0-7, B by 8-15: rows of 128 bytes in each of two slabs, their 16-byte pieces turned (the 128-byte swizzle)
    const float* src = (warp < 8 ? p.C : p.B) + (size_t)c.row0 * p.ld + group * N + (tid & 15) * 8;
    const uint32_t dst = (warp < 8 ? base : second) + ((tid & 15) >> 3) * (TILE / 2);
#pragma unroll 1
    for (int i0 = 0; i0 < 8; i0 += 4) {
      float v[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = ((tid & 255) >> 4) + (i0 + i) * 16;
        load8(src + (size_t)t * p.ld, t < c.tokens, v[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = ((tid & 255) >> 4) + (i0 + i) * 16;
        const float r = scale_of(most_of_row(v[i]));
        if ((tid & 15) == 0) (warp < 8 ? sm.inv_c : sm.inv_b)[t] = inverse_of(r);
        put_parts<0>(dst + t * 128 + (((tid & 7) ^ (t & 7)) << 4), TILE, v[i], &r);
      }
    }
    fence_proxy_async_smem();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem, 0), acc = tmem + 192;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  bool alive = true;

  const uint32_t one = elect_one();
  if (warp == 4) {
    issue<false>(one, SINGLES, 8, tmem, Operand{make_smem_desc(base), TILE >> 4, TILE >> 5, 2}, Operand{make_smem_desc(second), TILE >> 4, TILE >> 5, 2}, 128, 0u);
    commit_if(one, smem_u32(&sm.bars.cb_full));
  }
  __syncwarp();
  for (int j = warp - 8; warp >= 8 && j < units; j += 8) {       // while C B^T is made
    const Decays d = decays_of(p, c, (u0 + j) / p.per_head);
    double before = 1.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (i < (lane >> 3)) before *= d.block[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = 4 * lane + i;
      sm.a[j][t] = d.a[i];
      sm.dt[j][t] = d.dt[i];
      sm.upto[j][t] = (float)d.upto[i];
      sm.after[j][t] = (float)(d.after[i] * d.dt[i]);
      sm.pre[j][t] = (float)(before * d.upto[i]);
      if (lane == 0) sm.block[j][i] = (float)d.block[i];
    }
  }
  __syncthreads();
  if (warp < 8) {
    const int half = warp >> 2, t = (warp & 3) * 32 + lane, s0 = half * 64, own = warp & 3;       // own: t's block of 32
    const uint32_t cb = tmem + 384 + s0 + lanes;                   // C B^T, added up: this thread's 64 columns
    if ((alive = warp_wait(smem_u32(&sm.bars.cb_full), 0u, dead))) {
      tcgen05_fence_after();
#pragma unroll 1
      for (int q = 0; q < 64; q += 16) {
        uint32_t v[3][16];
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_ld16(tmem + i * 128 + s0 + q + lanes, v[i]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) v[0][i] = __float_as_uint(gathered(v[0][i], v[1][i], v[2][i]) * sm.inv_c[t] * sm.inv_b[s0 + q + i]);
        tmem_st16(cb + q, v[0]);
      }
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.bars.cb_read));
      alive = warp_wait(smem_u32(&sm.bars.cb_read), 0u, dead);     // the weights go where its parts were
      tcgen05_fence_after();
    }
    // The weight of token s for token t is a product over the blocks of 32 between them: up to t in its own, whole blocks, after s in its own.  Only within the same block it is
    // multiplied up token by token, from the last one on.  Blocks after t's are never looked at: the weights there are zero.  use(token, weights of 16 tokens)
    auto weights = [&](int j, auto use) {
#pragma unroll 1
      for (int b = 1; b >= 0; --b) {
        const int block = 2 * half + b;
        if (block > own) continue;
        float run = block < own ? sm.upto[j][t] : 1.f;
        for (int k = block + 1; k < own; ++k) run *= sm.block[j][k];
#pragma unroll 1
        for (int q = 32 * b + 16; q >= 32 * b; q -= 16) {
          uint32_t v[16];
          float w[16];
          tmem_ld16(cb + q, v);
          tmem_ld_wait();
          if (block < own) {
            const float* after = &sm.after[j][s0 + q];
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 f = *reinterpret_cast<const float4*>(after + i);
              w[i] = __uint_as_float(v[i]) * (run * f.x);
              w[i + 1] = __uint_as_float(v[i + 1]) * (run * f.y);
              w[i + 2] = __uint_as_float(v[i + 2]) * (run * f.z);
              w[i + 3] = __uint_as_float(v[i + 3]) * (run * f.w);
            }
          } else {
            const float* a = &sm.a[j][s0 + q];
            const float* dt = &sm.dt[j][s0 + q];
            const int last = lane - (q & 31);                      // the token itself
#pragma unroll
            for (int i = 14; i >= 0; i -= 2) {
              const float2 av = *reinterpret_cast<const float2*>(a + i), dv = *reinterpret_cast<const float2*>(dt + i);
              w[i + 1] = i + 1 <= last ? __uint_as_float(v[i + 1]) * (run * dv.y) : 0.f;
              run = i + 1 <= last ? run * av.y : run;
              w[i] = i <= last ? __uint_as_float(v[i]) * (run * dv.x) : 0.f;
              run = i <= last ? run * av.x : run;
            }
          }
          use(q, w);
        }
      }
    };
    {
      uint32_t w[8] = {};
#pragma unroll 1
      for (int q = 0; q < 64 && alive; q += 16)
        if (2 * half + (q >> 5) > own)
          for (int k = 0; k < 3; ++k) tmem_st8(tmem + k * 64 + (s0 + q) / 2 + lanes, w);
    }
    if (warp == 4) {
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
#pragma unroll 1
      for (int j = 0; alive && j < units; ++j) {
        const uint32_t parity = j & 1;
        if (!warp_wait(smem_u32(&sm.bars.s_full), parity, dead) || !warp_wait(smem_u32(&sm.bars.intra_read), parity ^ 1u, dead)) break;
        if (one) mbar_arrive(smem_u32(&sm.bars.inter_scaled));
        tcgen05_fence_after();
        issue<false>(one, PRODUCTS, 7, acc, Operand{make_smem_desc(base), TILE >> 4, TILE >> 5, 2}, Operand{make_smem_desc(ss), P * 128 >> 4, S_HALF >> 4, 2}, 64, 0u);
        commit_if(one, smem_u32(&sm.bars.inter_full));
        if (!warp_wait(smem_u32(&sm.bars.x_full), parity, dead) || !warp_wait(smem_u32(&sm.bars.inter_read), parity, dead) || !warp_wait(smem_u32(&sm.bars.w_full), parity, dead)) break;
        if (one) mbar_arrive(smem_u32(&sm.bars.intra_scaled));
        tcgen05_fence_after();
        issue<true>(one, PRODUCTS, 7, acc, Operand{tmem, 64, 32, 8}, Operand{make_smem_desc_mn(xs, UNIT), UNIT >> 4, 512, 128}, 64, 1u << 16);
        commit_if(one, smem_u32(&sm.bars.intra_full));
      }
      __syncwarp();
    } else
    for (int j = 0; j < units; ++j) {                              // (the two warps of a row meet at barriers whether alive or not)
      float most = 0.f;
      if (alive)
        weights(j, [&](int, const float* w) {
#pragma unroll
          for (int i = 0; i < 16; ++i) most = fmaxf(most, fabsf(w[i]));
        });
      if (own > 0) {
        sm.most_w[half][t] = most;
        asm volatile("bar.sync %0, 64;" ::"r"(2 + own) : "memory");
        most = fmaxf(most, sm.most_w[half ^ 1][t]);
        asm volatile("bar.sync %0, 64;" ::"r"(2 + own) : "memory");  // it is read
      }
      const float r = scale_of(most);
      if (alive && j > 0) {
        alive = warp_wait(smem_u32(&sm.bars.intra_full), (j - 1) & 1, dead);
        tcgen05_fence_after();
      }
      if (half == 0) sm.inv_w[j & 1][t] = inverse_of(r);           // (the outputs of the last unit but one are done: the last one's products waited for them)
      if (alive) {
        weights(j, [&](int q, const float* w) {
          uint32_t part[3][8];
#pragma unroll
          for (int i = 0; i < 8; ++i) split3(w[2 * i], w[2 * i + 1], r, r, part[0][i], part[1][i], part[2][i]);
#pragma unroll
          for (int k = 0; k < 3; ++k) tmem_st8(tmem + k * 64 + (s0 + q) / 2 + lanes, part[k]);
        });
        tmem_st_wait();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.bars.w_full));
      }
    }
  } else if (warp < 12) {
    const int t = tid - 256;                                       // token of the outputs
    int j = 0;
    for (; j < units && alive; ++j) {
      const uint32_t parity = j & 1;
      float y[P];
      const float dh = p.D[(u0 + j) / p.per_head];                 // D x, of x as it is
      const float* xrow = p.x + (size_t)(c.row0 + t) * p.ld + (u0 + j) * P;
#pragma unroll
      for (int q = 0; q < P; q += 8) {
        load8(xrow + q, t < c.tokens, y + q);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[q + i] *= dh;
      }
      if (!(alive = warp_wait(smem_u32(&sm.bars.inter_scaled), parity, dead) && warp_wait(smem_u32(&sm.bars.inter_full), parity, dead))) break;
      tcgen05_fence_after();
      const float pre = sm.pre[j][t], inv_c = sm.inv_c[t];
#pragma unroll
      for (int q = 0; q < P; q += 8) {
        uint32_t v[3][8];
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_ld8(acc + i * 64 + q + lanes, v[i]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) y[q + i] = fmaf(pre, gathered(v[0][i], v[1][i], v[2][i]) * inv_c * sm.inv_s[j & 1][q + i], y[q + i]);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.bars.inter_read));
      if (!(alive = warp_wait(smem_u32(&sm.bars.intra_scaled), parity, dead) && warp_wait(smem_u32(&sm.bars.intra_full), parity, dead))) break;
      tcgen05_fence_after();
      const float inv_w = sm.inv_w[j & 1][t];
      float* dst = p.o + (size_t)(c.row0 + t) * p.U * P + (u0 + j) * P;
#pragma unroll
      for (int q = 0; q < P; q += 8) {
        uint32_t v[3][8];
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_ld8(acc + i * 64 + q + lanes, v[i]);
        tmem_ld_wait();
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = y[q + i] + gathered(v[0][i], v[1][i], v[2][i]) * inv_w * sm.inv_x[q + i];
        if (q == P - 8) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sm.bars.intra_read));           // the scales are read, too
        }
        if (t < c.tokens) {
          *reinterpret_cast<float4*>(dst + q) = make_float4(f[0], f[1], f[2], f[3]);
          *reinterpret_cast<float4*>(dst + q + 4) = make_float4(f[4], f[5], f[6], f[7]);
        }
      }
    }
    for (; j < units; ++j)                                         // a wait ran out: these outputs will not be
      if (t < c.tokens)
        for (int i = 0; i < P; ++i) p.o[(size_t)(c.row0 + t) * p.U * P + (u0 + j) * P + i] = NAN;
  } else {
    const int th = tid - 384;
    float v[8][8];
    auto get_state = [&](int j) {                                  // rows th / 16 + 8 i of the unit's columns, 8 rows of the state each
      const float* src = p.states + ((size_t)blockIdx.x * p.U + u0 + j) * P * N + th * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) load8(src + i * 1024, true, v[i]);
    };
    auto put_state = [&](int j) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = (th >> 4) + i * 8;
        const float scale = scale_of(most_of_row(v[i]));
        if ((th & 15) == 0) sm.inv_s[j & 1][r] = inverse_of(scale);
        put_parts<0>(ss + ((th & 15) >> 3) * S_HALF + r * 128 + (((th & 7) ^ (r & 7)) << 4), P * 128, v[i], &scale);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.bars.s_full));
    };
    auto get_x = [&](int j) {                                      // tokens th / 8 + 16 i, columns 8 (th % 8) ..
      const float* src = p.x + (size_t)c.row0 * p.ld + (u0 + j) * P + (th & 7) * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = (th >> 3) + i * 16;
        load8(src + (size_t)t * p.ld, t < c.tokens, v[i]);
      }
    };
    float most[8];
    auto scales_of_x = [&]() {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        most[e] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) most[e] = fmaxf(most[e], fabsf(v[i][e]));
        most[e] = fmaxf(most[e], __shfl_xor_sync(0xffffffffu, most[e], 8));
        most[e] = fmaxf(most[e], __shfl_xor_sync(0xffffffffu, most[e], 16));
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");               // the last unit's are read
      if (lane < 8) {
#pragma unroll
        for (int e = 0; e < 8; e += 4) *reinterpret_cast<float4*>(&sm.most_x[warp - 12][lane * 8 + e]) = make_float4(most[e], most[e + 1], most[e + 2], most[e + 3]);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      scales_of(sm.most_x, (lane & 7) * 8, most);
    };
    get_state(0);
    alive = warp_wait(smem_u32(&sm.bars.cb_full), 0u, dead) && warp_wait(smem_u32(&sm.bars.cb_read), 0u, dead);       // B and C B^T are read
    for (int j = 0; j < units; ++j) {                              // (the four warps meet at barriers whether alive or not)
      const uint32_t parity = j & 1;
      if (alive) put_state(j);                                     // C S of the last unit is done: its outputs were waited for
      get_x(j);
      scales_of_x();
      if (alive && j > 0) alive = warp_wait(smem_u32(&sm.bars.intra_read), parity ^ 1u, dead);       // the last unit's x is read, by its product and by its outputs
      if (alive) {
        if (th < 8) {
#pragma unroll
          for (int e = 0; e < 8; ++e) sm.inv_x[th * 8 + e] = inverse_of(most[e]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = (th >> 3) + i * 16;
          put_parts<1>(xs + t * 128 + (((th & 7) ^ (t & 7)) << 4), UNIT, v[i], most);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.bars.x_full));
      }
      if (j + 1 < units) get_state(j + 1);
      if (alive) alive = warp_wait(smem_u32(&sm.bars.inter_full), parity, dead);           // the state's place is free
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (*dead) {
    if (warp == 4) {                                               // products in flight end before shared memory and TMEM are given back
      if (one) atomicAdd_system(p.timeouts, 1);
      commit_if(one, smem_u32(&sm.bars.drain));
      wait_in_flight(smem_u32(&sm.bars.drain), 0u);
    }
    __syncthreads();
  }
  if (warp == 4) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

long long round16(long long n) { return (n + 15) / 16 * 16; }
// of `longs` portions of SHORT tokens and more, `rows` tokens together
long long slots_of(long long rows, long long longs, long long chunks) { return std::min(longs * chunks, (rows + longs * (L - 1)) / L); }
long long bytes_of(long long slots, long long longs, int H, long long U) { return slots * U * (P * N * 4 + 12) + longs * U * P * N * 4 + round16(4 * longs * H) + 16; }
int longs_of(int rows, int nseg) { return std::max(1, std::min(nseg, rows / SHORT)); }         // at most

}  // namespace

extern "C" int lia_ssd_chunk_rows() { return SHORT; }

/* Bytes of workspace for taking `chunks` chunks of every portion at a time (see lia_b200.h); 0: the step goes token by token */
extern "C" long long lia_ssd_workspace(int rows, int nseg, int H, int G, int Ns, int vdim, int chunks) {
  if (Ns != N || vdim <= 0 || vdim % P || nseg <= 0 || nseg > 65535 || H <= 0 || G <= 0 || H % G || chunks <= 0 || rows - nseg + 1 < 2 * L) return 0;
  const long long U = (long long)H * (vdim / P);
  if (U > 8191) return 0;
  const int longs = longs_of(rows, nseg);
  return bytes_of(slots_of(rows, longs, chunks), longs, H, U);
}

// `longs` portions of SHORT tokens and more, `long_rows` tokens together and `longest` at most; the others `others`
static int scan_chunks(const float* B, const float* C, const float* x, int ld, const float* gates, const float* D, float* state_S, const int* segs, int nseg, int longs, int long_rows,
                       int longest, int others, int H, int G, int Ns, int vdim, float* o, void* ws, long long ws_bytes, int chunks, cudaStream_t stream) {
  const long long need = lia_ssd_workspace(long_rows, longs, H, G, Ns, vdim, chunks);
  LIA_CHECK_ARG(need > 0 && nseg > 0 && nseg <= 65535, "lia_ssd_scan_chunks: bad shape nseg=%d rows=%d H=%d G=%d N=%d vdim=%d", nseg, long_rows, H, G, Ns, vdim);
  LIA_CHECK_ARG(ws_bytes >= need, "lia_ssd_scan_chunks: the workspace holds %lld of %lld bytes", ws_bytes, need);
  const uintptr_t all = reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(state_S) |
                        reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(ws);
  LIA_CHECK_ARG(all % 16 == 0 && ld % 4 == 0, "lia_ssd_scan_chunks: rows are not whole 16-byte vectors");
  const int U = H * (vdim / P), per_group = U / G, sms = lia_sm_count();
  const long long slots = slots_of(long_rows, longs, chunks);
  LIA_CHECK_ARG(slots < (1ll << 31), "lia_ssd_scan_chunks: too many rows");
  SsdArgs p{B, C, x, ld, gates, D, state_S, segs, nseg, H, G, U, vdim / P, o};
  p.states = reinterpret_cast<float*>(ws);
  p.after = p.states + slots * U * P * N;
  p.slots = (int)slots;
  p.longs = longs;
  p.totals = reinterpret_cast<float2*>(p.after + (long long)longs * U * P * N);
  p.bad = reinterpret_cast<int*>(p.totals + slots * U);
  p.flags = p.bad + slots * U;
  p.timeouts = lia_timeout_word();
  LIA_CHECK_ARG(p.timeouts != nullptr, "lia_ssd_scan_chunks: no host memory for the count of timeouts");
  // B and C are split once per CTA: few CTAs with many units each, as long as there is one for every SM
  p.split = (per_group + MAX_UNITS - 1) / MAX_UNITS;
  while (p.split < per_group && 2 * slots * G * p.split <= sms) p.split *= 2;
  p.per_cta = (per_group + p.split - 1) / p.split;
  LIA_CHECK_ARG((long long)G * p.split <= 65535, "lia_ssd_scan_chunks: too many groups (%d)", G);
  LIA_CUDA(cudaFuncSetAttribute(ssd_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_BYTES));
  LIA_CUDA(cudaFuncSetAttribute(ssd_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_BYTES));
  p.span = chunks * L;
  for (int tok0 = 0; tok0 < longest; tok0 += p.span) {
    p.tok0 = tok0;
    const dim3 grid((unsigned)slots, (unsigned)(G * p.split));
    lia_launch(ssd_states_kernel, grid, dim3(ST_THREADS), ST_BYTES, stream, p);
    LIA_LAUNCH_CHECK();
    lia_launch(ssd_carry_kernel, dim3((unsigned)U * 8, (unsigned)longs), dim3(CARRY), 0, stream, p);
    LIA_LAUNCH_CHECK();
    lia_launch(ssd_outputs_kernel, grid, dim3(OUT_THREADS), OUT_BYTES, stream, p);
    LIA_LAUNCH_CHECK();
    const int rc = ssd_scan_tokens(B, C, x, ld, gates, D, state_S, segs, tok0, p.span, SHORT, longs, p.flags, p.after, others == 1, nseg, H, G, Ns, vdim, o, stream);
    if (rc != LIA_OK) return rc;
  }
  return LIA_OK;
}

/* see lia_b200.h */
extern "C" int lia_ssd_scan_chunks(const float* B, const float* C, const float* x, int ld, const float* gates, const float* D, float* state_S, const int* segs, int nseg,
                                   int rows, int H, int G, int Ns, int vdim, float* o, void* ws, long long ws_bytes, int chunks, lia_stream_t stream) {
  LIA_CHECK_ARG(B && C && x && gates && D && state_S && segs && o && ws, "lia_ssd_scan_chunks: null pointer");
  LIA_CHECK_ARG(lia_ssd_workspace(rows, nseg, H, G, Ns, vdim, chunks) > 0, "lia_ssd_scan_chunks: bad shape nseg=%d rows=%d H=%d G=%d N=%d vdim=%d", nseg, rows, H, G, Ns, vdim);
  return scan_chunks(B, C, x, ld, gates, D, state_S, segs, nseg, longs_of(rows, nseg), rows, rows, SHORT - 1, H, G, Ns, vdim, o, ws, ws_bytes, chunks, reinterpret_cast<cudaStream_t>(stream));
}
extern "C" int lia_ssd_scan_long(const float* B, const float* C, const float* x, int ld, const float* gates, const float* D, float* state_S, const int* segs, int nseg,
                                 int longs, int long_rows, int longest, int others, int H, int G, int Ns, int vdim, float* o, void* ws, long long ws_bytes, int chunks,
                                 lia_stream_t stream) {
  LIA_CHECK_ARG(B && C && x && gates && D && state_S && segs && o && ws, "lia_ssd_scan_long: null pointer");
  LIA_CHECK_ARG(longs > 0 && longs <= nseg && longest >= SHORT && longest <= long_rows && (long long)longs * SHORT <= long_rows && others >= 0 && others < SHORT && chunks > 0,
                "lia_ssd_scan_long: %d portions of %d tokens, the longest one's %d", longs, long_rows, longest);
  return scan_chunks(B, C, x, ld, gates, D, state_S, segs, nseg, longs, long_rows, longest, others, H, G, Ns, vdim, o, ws, ws_bytes, chunks, reinterpret_cast<cudaStream_t>(stream));
}
