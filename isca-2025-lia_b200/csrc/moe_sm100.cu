// Projections of a mixture's experts, each over its own rows, as ONE tcgen05 launch per projection (bf16 weights and rows).
//
//   up:    mid[row]  = act(a[row] . Wup_e^T), or act(gate) * up with both sums in fp32 in one tile -- the plan's rows in their order
//   down:  out[row]  = a[row] . Wdown_e^T in the plan's order (bf16), or ypair[pair] = wt[pair] * (...) per pair (fp32)
//
// The plan (lia_moe_plan_rows with tiles of 128 rows) lists the experts' row tiles one after the other, every tile of one expert; the grid walks
// (row tile, column tile) pairs, column tiles of one row tile side by side.  Nothing about the plan is known to the host: the number of tiles
// in use is counted from tile_expert, so there is no round trip and a step with experts can be captured.
//
// One persistent CTA per SM, 256 threads: warp 0 loads by TMA (128-byte swizzle; 16 KB of rows and 32 KB of weights per stage, 4 stages), one lane
// of warp 1 issues tcgen05.mma (128 x 256 x 16), warps 4-7 drain one of two TMEM accumulators of 256 columns while the other is filled.
// Gated: the 256 weight rows of a tile are 128 gate and 128 up rows.  Bound: the weights' bytes up to about 128 rows per expert, then the
// tensor cores.  2048 rows of 2048 channels, 16 gated experts of 1408, 2 chosen: 95 us up (4.7e10 FLOPs, 500 TFLOP/s) and 34 us down (700); the whole
// feed-forward 742 us with one launch per expert and projection, each a quarter full, a host round trip and two more passes over bf16 sums
// -> 178 us.  150 rows, whose experts' weights (277 MB) are the bound: 903 us on the CUDA cores -> 113 us.
//
// One accumulator runs over the whole of K, and the tensor cores cut its sums off below the 24th bit: against 64 bits the fp32 outputs of the down projection alone are
// off by 8e-7, 1.6e-6, 3.3e-6 at width 1024, 2048, 4096 (FMA chains: 2.8e-7, 4.2e-7, 6.4e-7).  Their inputs are bf16 numbers, each rounded by up to 2^-9: the feed-forward
// is off by 0.00165 either way.
//
// Every wait is bounded: a barrier that does not come within the limit raises a flag in shared memory, all roles leave, what the CTA still owed becomes NaN, loads
// and products in flight are waited for, and a word in host memory counts the CTA (lia_moe_timeouts_seen(), which the engine asks before each step).
#include <cuda.h>

#include <mutex>

#include "act.cuh"
#include "common.cuh"
#include "umma.cuh"

namespace {

constexpr int ROWS = 128, KB = 64;
// COLS weight rows per tile: 256, or 128 where that fills the last round of tiles better
template <int COLS> struct Shape {
  static constexpr int STAGES = COLS == 256 ? 4 : 6;
  static constexpr int A_BYTES = ROWS * KB * 2, B_BYTES = COLS * KB * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGING = 4 * 4096;                         // 32 rows of 128 bytes per epilogue warp
  static constexpr int BARS = STAGES * STAGE_BYTES + STAGING;
  static constexpr int SMEM = BARS + (2 * STAGES + 5) * 8 + 16 + 1024;
};
struct MoeArgs {
  const int* perm;
  const int* tile_expert;
  const float* wt;
  void* out;
  long long out_ld;
  int n_tiles, n_real, N, n_rows_w, k_blocks, act, weigh_in;       // N: output columns; n_rows_w: weight rows of an expert
  float p0, p1;
  int* timeouts;                                                   // in host memory
};

enum { UP, UP_GATED, DOWN_PLAN, DOWN_PAIR };

template <int MODE, int COLS>
__global__ void __launch_bounds__(256, 1) moe_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const MoeArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr bool GATED = MODE == UP_GATED;
  constexpr int OUT_COLS = GATED ? COLS / 2 : COLS;                // output columns of a tile
  constexpr int STAGES = Shape<COLS>::STAGES, A_BYTES = Shape<COLS>::A_BYTES, B_BYTES = Shape<COLS>::B_BYTES, STAGE_BYTES = Shape<COLS>::STAGE_BYTES,
                BARS = Shape<COLS>::BARS;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + BARS;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + BARS + (2 * STAGES + 5) * 8);
  volatile int* dead = reinterpret_cast<volatile int*>(smem_gen + BARS + (2 * STAGES + 5) * 8 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
    *dead = 0;
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 4);
    }
    mbar_init(drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_ptr)), "r"(2u * COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // row tiles in use: those of experts that have weights (they come first)
  int used = 0;
  for (int t0 = 0; t0 < p.n_tiles; t0 += 256) {
    const int t = t0 + (int)threadIdx.x;
    const int e = t < p.n_tiles ? p.tile_expert[t] : -1;
    used += __syncthreads_count(e >= 0 && e < p.n_real);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  const int col_tiles = (p.N + OUT_COLS - 1) / OUT_COLS, total = used * col_tiles;
  int issued = 0;                                                  // loads of the producer's lane

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (int u = blockIdx.x; u < total && alive; u += gridDim.x) {
        const int tm = u / col_tiles, tn = u - tm * col_tiles;
        const int e = p.tile_expert[tm];
        const int row_w = e * p.n_rows_w + tn * OUT_COLS;
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!(alive = wait_for(empty_bar(stage), phase ^ 1u, dead))) break;
          const uint32_t sa = smem_base + stage * STAGE_BYTES, sb = sa + A_BYTES;
          mbar_expect_tx(full_bar(stage), STAGE_BYTES);
          tma_load_2d(sa, &tmA, kb * KB, tm * ROWS, full_bar(stage));
          tma_load_2d(sb, &tmB, kb * KB, row_w, full_bar(stage));
          tma_load_2d(sb + B_BYTES / 2, &tmB, kb * KB, GATED ? row_w + p.N : row_w + COLS / 2, full_bar(stage));
          ++issued;
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc(ROWS, COLS);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool alive = true;
      for (int u = blockIdx.x; u < total && alive; u += gridDim.x) {
        if (!(alive = wait_for(tempty_bar(acc), acc_phase ^ 1u, dead))) break;
        tcgen05_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(acc * COLS);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!(alive = wait_for(full_bar(stage), phase, dead))) break;
          tcgen05_fence_after();
          const uint32_t sa = smem_base + stage * STAGE_BYTES;
          const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + A_BYTES);
#pragma unroll
          for (int k = 0; k < KB / 16; ++k) tcgen05_mma_f16(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
          tcgen05_commit(empty_bar(stage));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!alive) break;
        tcgen05_commit(tfull_bar(acc));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (warp >= 4) {
    const int ew = warp - 4;
    const uint32_t stg = smem_base + STAGES * STAGE_BYTES + ew * 4096;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool alive = true;
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
      const int tm = u / col_tiles, tn = u - tm * col_tiles;
      const int row0 = tm * ROWS + ew * 32;                        // of this warp
      const int pair = p.perm[row0 + lane];
      const float w = (pair >= 0 && ((MODE == DOWN_PAIR && p.wt != nullptr) || ((MODE == UP || GATED) && p.weigh_in))) ? p.wt[pair] : 1.0f;
      alive = __all_sync(0xffffffffu, alive && wait_for(tfull_bar(acc), acc_phase, dead));
      if (!alive) {                                                // these outputs will not be: NaN, so that nobody takes them for some
        for (int r = 0; r < 32; ++r) {
          const int to = MODE == DOWN_PAIR ? __shfl_sync(0xffffffffu, pair, r) : row0 + r;
          for (int col = tn * OUT_COLS + lane; to >= 0 && col < min(p.N, (tn + 1) * OUT_COLS); col += 32) {
            if constexpr (MODE == DOWN_PAIR) reinterpret_cast<float*>(p.out)[(size_t)to * p.out_ld + col] = NAN;
            else reinterpret_cast<bf16*>(p.out)[(size_t)to * p.out_ld + col] = __float2bfloat16_rn(NAN);
          }
        }
        continue;
      }
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t)(acc * COLS) + ((uint32_t)(ew * 32) << 16);
      constexpr int SLAB = MODE == DOWN_PAIR ? 32 : 64;            // columns of 128 bytes
#pragma unroll 1
      for (int c0 = 0; c0 < OUT_COLS; c0 += SLAB) {
#pragma unroll
        for (int half = 0; half < SLAB / 32; ++half) {
          uint32_t v[32];
          float f[32];
          tmem_ld32(taddr + c0 + half * 32, v);
          if constexpr (GATED) {
            uint32_t v2[32];
            tmem_ld32(taddr + OUT_COLS + c0 + half * 32, v2);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = gated_apply(w * __uint_as_float(v[i]), w * __uint_as_float(v2[i]), p.act, p.p0, p.p1);
          } else {
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = MODE == UP ? act_apply(w * __uint_as_float(v[i]), p.act) : w * __uint_as_float(v[i]);
          }
          // 16-byte chunks of the warp's rows, each row's chunks turned by the row so that neither side of the transposition collides
          constexpr int CHUNKS = MODE == DOWN_PAIR ? 8 : 4;
#pragma unroll
          for (int j = 0; j < CHUNKS; ++j) {
            const int chunk = half * 4 + j;
            uint4 q;
            if constexpr (MODE == DOWN_PAIR) q = make_uint4(__float_as_uint(f[4 * j]), __float_as_uint(f[4 * j + 1]), __float_as_uint(f[4 * j + 2]), __float_as_uint(f[4 * j + 3]));
            else q = pack8(f + 8 * j);
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(stg + lane * 128 + ((chunk ^ (lane & 7)) << 4)), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
          }
        }
        if (c0 + SLAB >= OUT_COLS) {                               // the accumulator is read: back to the MMA warp
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(tempty_bar(acc));
        } else {
          __syncwarp();
        }
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int r = it * 4 + (lane >> 3), chunk = lane & 7;
          uint4 q;
          asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "r"(stg + r * 128 + ((chunk ^ (r & 7)) << 4)));
          const int col = tn * OUT_COLS + c0 + chunk * (MODE == DOWN_PAIR ? 4 : 8);
          const int to = MODE == DOWN_PAIR ? __shfl_sync(0xffffffffu, pair, r) : row0 + r;
          if (col < p.N && to >= 0) {
            if constexpr (MODE == DOWN_PAIR) *reinterpret_cast<uint4*>(reinterpret_cast<float*>(p.out) + (size_t)to * p.out_ld + col) = q;
            else *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.out) + (size_t)to * p.out_ld + col) = q;
          }
        }
        __syncwarp();
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (*dead) {                                                     // loads and products in flight end before shared memory and TMEM are given back
    if (threadIdx.x == 0) {
      atomicAdd_system(p.timeouts, 1);
      for (int i = 0; i < STAGES && i < issued; ++i) {
        const int n = issued - 1 - i;
        wait_in_flight(full_bar(n % STAGES), (uint32_t)(n / STAGES) & 1u);
      }
    }
    if (warp == 1 && lane == 0) {
      tcgen05_commit(drain_bar);
      wait_in_flight(drain_bar, 0u);
    }
    __syncthreads();
  }
  if (warp == 2) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2u * COLS) : "memory");
  }
}

template <int MODE, int COLS> int launch_as(const CUtensorMap& tmA, const CUtensorMap& tmB, const MoeArgs& a, long long tiles, cudaStream_t stream) {
  LIA_CUDA(cudaFuncSetAttribute(moe_tc_kernel<MODE, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<COLS>::SMEM));
  const int sms = lia_sm_count();
  lia_launch(moe_tc_kernel<MODE, COLS>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(256), Shape<COLS>::SMEM, stream, tmA, tmB, a);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

// What a tile takes is its operands' way from L2 (13 TB/s for all SMs; the tensor cores alone would take half that time): 384 rows of 128 bytes a block of K for the wide tile, 256 for the
// narrow one, which is taken where its rounds over the SMs come out shorter or alike.  2048 rows, 16 gated experts of 1408 columns, K = 2048, at most 48 row tiles: 4 wide rounds 55 us,
// 8 narrow ones 73; on one row tile each, 2 and 3 rounds: 79 and 62 us.
template <int MODE> int launch(const void* W, uint64_t w_rows, int K, const CUtensorMap& tmA, const MoeArgs& a, cudaStream_t stream) {
  const int per_wide = MODE == UP_GATED ? 128 : 256, sms = lia_sm_count();
  const long long wide = (long long)a.n_tiles * ((a.N + per_wide - 1) / per_wide), narrow = (long long)a.n_tiles * ((a.N + per_wide / 2 - 1) / (per_wide / 2));
  const bool use_narrow = ((narrow + sms - 1) / sms) * 2 <= ((wide + sms - 1) / sms) * 3;
  CUtensorMap tmB;
  const int rc = lia_make_tmap_2d(&tmB, W, w_rows, K, K, use_narrow ? 64 : 128);
  if (rc != LIA_OK) return rc;
  return use_narrow ? launch_as<MODE, 128>(tmA, tmB, a, narrow, stream) : launch_as<MODE, 256>(tmA, tmB, a, wide, stream);
}

}  // namespace

extern "C" int lia_moe_tc_rows(void) { return ROWS; }

// The word that counts CTAs whose wait ran out: host memory that every GPU can write, allocated with the first launch and kept.
static int* timeout_word(bool make) {
  static std::mutex m;
  static int* word = nullptr;
  std::lock_guard<std::mutex> lock(m);
  if (word == nullptr && make) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;     // the first launch may be part of a capture
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      word = static_cast<int*>(p);
      *word = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  return word;
}
int* lia_timeout_word() { return timeout_word(true); }             // for the kernels of other files

/* CTAs of the tcgen05 kernels with bounded waits (lia_moe_gemm_tc, lia_ssd_scan_chunks, prompts of lia_window_attn_mma and lia_latent_attn_expanded) that gave up one, as far as launches have ended, since the library was loaded */
extern "C" int lia_moe_timeouts_seen(void) {
  const volatile int* word = timeout_word(false);
  return word ? *word : 0;
}

/* the same after all launches (synchronises) */
extern "C" int lia_moe_timeouts(void) {
  LIA_CUDA(cudaDeviceSynchronize());
  return lia_moe_timeouts_seen();
}

extern "C" int lia_moe_gemm_tc(const void* A, const void* W, void* C, int c_f32, const int* perm, const int* tile_expert, int n_tiles, const float* wt, int N,
                               int K, int E, int up, int act, int gated, float p0, float p1, int weigh_in, lia_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LIA_CHECK_ARG(A && W && C && perm && tile_expert && n_tiles > 0 && N > 0 && K > 0 && E > 0, "lia_moe_gemm_tc: bad arguments");
  LIA_CHECK_ARG(N % 8 == 0 && K % 8 == 0, "lia_moe_gemm_tc: K and N must be multiples of 8 (got K=%d N=%d)", K, N);
  LIA_CHECK_ARG((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(C)) % 16 == 0, "lia_moe_gemm_tc: operands must be 16-byte aligned");
  LIA_CHECK_ARG(!gated || up, "lia_moe_gemm_tc: only the up projection can be gated");
  LIA_CHECK_ARG(act != LIA_ACT_CLAMPED_SWISH || (gated && p0 > 0.f), "lia_moe_gemm_tc: the clamped activation needs the gated form and a positive limit");
  LIA_CHECK_ARG(!(up && c_f32) && (wt || (up ? !weigh_in : (!c_f32 || weigh_in))), "lia_moe_gemm_tc: the up projection writes bf16; routing weights are missing");
  const int rows_w = gated ? 2 * N : N;
  LIA_CHECK_ARG((long long)E * rows_w < (1ll << 31) && (long long)n_tiles * ROWS < (1ll << 31) && (long long)n_tiles * ((N + 63) / 64) < (1ll << 31), "lia_moe_gemm_tc: too large");
  CUtensorMap tmA;
  const int rc = lia_make_tmap_2d(&tmA, A, (uint64_t)n_tiles * ROWS, K, K, ROWS);
  if (rc != LIA_OK) return rc;
  const uint64_t w_rows = (uint64_t)E * rows_w;
  MoeArgs a{perm, tile_expert, wt, C, N, n_tiles, E, N, rows_w, (K + KB - 1) / KB, act, weigh_in, p0, p1, timeout_word(true)};
  LIA_CHECK_ARG(a.timeouts != nullptr, "lia_moe_gemm_tc: no host memory for the count of timeouts");
  if (up) return gated ? launch<UP_GATED>(W, w_rows, K, tmA, a, stream) : launch<UP>(W, w_rows, K, tmA, a, stream);
  if (!c_f32) return launch<DOWN_PLAN>(W, w_rows, K, tmA, a, stream);
  if (weigh_in) a.wt = nullptr;
  return launch<DOWN_PAIR>(W, w_rows, K, tmA, a, stream);
}
