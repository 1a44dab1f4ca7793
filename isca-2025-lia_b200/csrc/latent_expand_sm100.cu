// Latents to keys and values (latent_attn_mma.cu) on tcgen05: up to 16 ranges of cached bf16 rows times bf16 weights, the fp32 sums as three bf16 parts.
//
// A CTA keeps 128 rows (all of K, up to 512) in shared memory and takes 32 columns of the weights after the other, so that only those are fetched again.  The tensor cores cut sums off below the
// 24th bit, towards zero, by as much of the sum for every instruction of a chain: each half of K has eight accumulators, which take every eighth instruction (two each at K = 512, as many as the
// kernel replaced; four put attention over the results off by 1.10 times as much), and all are added in fp32.  One half's are drained while the other's are filled.
// Bound: the products, 32 of 42 clocks per 128 x 32 sums, beside the parts' way out.  2048 latents of 512 to 16 heads of 128 (50 MB of parts): 67 us on mma.sync -> 29; 64 latents 17 -> 6.
// Waits are bounded: a CTA that gives up leaves NaN and counts itself (lia_moe_timeouts_seen()).
#include <algorithm>

#include "mma.cuh"
#include "umma.cuh"

int* lia_timeout_word();                                           // moe_sm100.cu

namespace {

constexpr int ROWS = 128, COLS = 32, MAX_K = 512, STAGES = 3, ACCS = 8, MAX_RANGES = 16, THREADS = 320;
struct ExpandArgs {
  int n, tiles, K, part, col_tiles;
  int row0[MAX_RANGES], rows[MAX_RANGES], tile0[MAX_RANGES], out0[MAX_RANGES];       // a range's first row in the map, its rows, first tile and first row of the result
  bf16* C;
  long long ldc;
};
struct Tail {
  uint64_t a_full, w_full[STAGES], w_empty[STAGES], acc_full[2][2], acc_empty[2], drain;      // acc_full: of a half, for either group of warps
  uint32_t tmem;
  int dead, issued;                                                // issued: tiles of weights asked for
};
int smem_of(int K) { return K / 64 * (ROWS + STAGES * COLS) * 128 + (int)sizeof(Tail) + 1024; }

__global__ void __launch_bounds__(THREADS, 1) latent_expand_kernel(const __grid_constant__ CUtensorMap rows_map, const __grid_constant__ CUtensorMap w_map, const __grid_constant__ ExpandArgs p,
                                                                    int* timeouts) {
  extern __shared__ uint8_t raw[];
  const int slabs = p.K / 64, first = (slabs + 1) / 2;             // slabs of the first half
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u, ws = base + slabs * ROWS * 128, w_bytes = slabs * COLS * 128;
  Tail& sm = *reinterpret_cast<Tail*>(raw + (base - smem_u32(raw)) + slabs * (ROWS + STAGES * COLS) * 128);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  volatile int* dead = &sm.dead;
  if (tid == 0) {
    sm.dead = sm.issued = 0;
    asm volatile("prefetch.tensormap [%0];" ::"l"(&rows_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w_map) : "memory");
    mbar_init(smem_u32(&sm.a_full), 1);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&sm.w_full[i]), 1);
      mbar_init(smem_u32(&sm.w_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      for (int k = 0; k < 2; ++k) mbar_init(smem_u32(&sm.acc_full[i][k]), 1);
      mbar_init(smem_u32(&sm.acc_empty[i]), 4);
    }
    mbar_init(smem_u32(&sm.drain), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem, 0);
  pdl_launch_dependents();
  const int tile = blockIdx.x % p.tiles, group = blockIdx.x / p.tiles, groups = gridDim.x / p.tiles;
  const int c0 = p.col_tiles * group / groups, c1 = p.col_tiles * (group + 1) / groups;
  int i = 0;
  while (i + 1 < p.n && tile >= p.tile0[i + 1]) ++i;
  const int skip = (tile - p.tile0[i]) * ROWS;
  pdl_wait();

  if (warp == 8) {
    const uint32_t one = elect_one();
    if (one) {
      mbar_expect_tx(smem_u32(&sm.a_full), slabs * ROWS * 128);
      for (int k = 0; k < slabs; ++k) tma_load_2d(base + k * ROWS * 128, &rows_map, k * 64, p.row0[i] + skip, smem_u32(&sm.a_full));
    }
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
      const int n = c - c0, st = n % STAGES;
      if (!warp_wait(smem_u32(&sm.w_empty[st]), (uint32_t)(n / STAGES & 1) ^ 1u, dead)) break;
      if (!one) continue;
      sm.issued = n + 1;
      mbar_expect_tx(smem_u32(&sm.w_full[st]), w_bytes);
      for (int k = 0; k < slabs; ++k) tma_load_2d(ws + st * w_bytes + k * COLS * 128, &w_map, k * 64, c * COLS, smem_u32(&sm.w_full[st]));
    }
  } else if (warp == 9) {
    const uint32_t one = elect_one();
    constexpr uint32_t idesc = make_idesc(ROWS, COLS);
    const uint64_t a_desc = make_smem_desc(base), w_desc = make_smem_desc(ws);
    bool alive = warp_wait(smem_u32(&sm.a_full), 0u, dead);
#pragma unroll 1
    for (int c = c0; alive && c < c1; ++c) {
      const int n = c - c0, st = n % STAGES;
      if (!(alive = warp_wait(smem_u32(&sm.w_full[st]), n / STAGES & 1, dead))) break;
      uint64_t a = a_desc, w = w_desc + (uint32_t)(st * w_bytes >> 4);
#pragma unroll 1
      for (int half = 0; alive && half < 2 && half * first < slabs; ++half) {
        if (!(alive = warp_wait(smem_u32(&sm.acc_empty[half]), (uint32_t)(n & 1) ^ 1u, dead))) break;
        tcgen05_fence_after();
        const int count = half ? slabs - first : first;
#pragma unroll 1
        for (int k = 0; k < count; ++k, a += ROWS * 128 >> 4, w += COLS * 128 >> 4) {
          const uint32_t d = tmem + half * (ACCS * COLS) + (k & 1) * (4 * COLS);
#pragma unroll
          for (int q = 0; q < 4; ++q) mma_if(one, d + q * COLS, a + 2 * q, w + 2 * q, idesc, k > 1);
        }
        if ((half + 1) * first >= slabs) commit_if(one, smem_u32(&sm.w_empty[st]));
        commit_if(one, smem_u32(&sm.acc_full[half][n & 1]));
      }
    }
  } else {
    const int group_of_four = warp >> 2, r = (warp & 3) * 32 + lane;
    const bool live = skip + r < p.rows[i];
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    bf16* row = p.C + (size_t)(p.out0[i] + skip + r) * p.ldc;
    bool alive = true;                                             // (the whole warp's, as the waits are: a lane without a row goes round with the others)
#pragma unroll 1
    for (int c = c0 + group_of_four; c < c1; c += 2) {
      const int n = c - c0;
      float sum[COLS];
#pragma unroll
      for (int e = 0; e < COLS; ++e) sum[e] = 0.f;
#pragma unroll 1
      for (int half = 0; half < 2 && half * first < slabs; ++half) {
        alive = alive && warp_wait(smem_u32(&sm.acc_full[half][n & 1]), n >> 1 & 1, dead);
        tcgen05_fence_after();
        const int accs = min(ACCS, 4 * (half ? slabs - first : first));
#pragma unroll 1
        for (int q = 0; q < accs; q += 4) {                        // four together, and the fours in turn
          uint32_t u[4][COLS / 2];
#pragma unroll
          for (int e0 = 0; e0 < COLS; e0 += COLS / 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k) tmem_ld16(tmem + half * (ACCS * COLS) + (q + k) * COLS + e0 + lanes, u[k]);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < COLS / 2; ++e) sum[e0 + e] += (__uint_as_float(u[0][e]) + __uint_as_float(u[1][e])) + (__uint_as_float(u[2][e]) + __uint_as_float(u[3][e]));
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.acc_empty[half]));
      }
      if (!live) continue;
      const int col = c * COLS;
      bf16* out = row + (size_t)(col / p.part) * 3 * p.part + col % p.part;
#pragma unroll
      for (int e = 0; e < COLS; e += 8) {
        uint32_t part[3][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!alive) sum[e + 2 * k] = sum[e + 2 * k + 1] = NAN;
          split3(sum[e + 2 * k], sum[e + 2 * k + 1], part[0][k], part[1][k], part[2][k]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(out + (size_t)k * p.part + e) = make_uint4(part[k][0], part[k][1], part[k][2], part[k][3]);
      }
    }
  }
  tcgen05_fence_before();
  if (__syncthreads_or(*dead)) {                                   // products and loads in flight end before shared memory and TMEM are given back
    if (tid == 0) atomicAdd_system(timeouts, 1);
    if (warp == 9) {
      commit_if(elect_one(), smem_u32(&sm.drain));
      wait_in_flight(smem_u32(&sm.drain), 0u);
      wait_in_flight(smem_u32(&sm.a_full), 0u);
      for (int n = max(0, sm.issued - STAGES); n < sm.issued; ++n) wait_in_flight(smem_u32(&sm.w_full[n % STAGES]), n / STAGES & 1);
    }
    __syncthreads();
  }
  if (warp == 9) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

}  // namespace

// 1: latent_expand takes these latents and weights
bool latent_expand_takes(long long slot_stride, int D, int K, int N, int part) { return K % 64 == 0 && K <= MAX_K && N % COLS == 0 && part % COLS == 0 && slot_stride % D == 0 && D % 8 == 0; }

// C [rows of all ranges][N / part][3][part] of the rows first[i] .. first[i] + rows[i] - 1 of `cache` [.][D], of which the first K numbers count, and W [N][K]
int latent_expand(const bf16* cache, int D, const long long* first, const int* rows, int n, const bf16* W, bf16* C, long long ldc, int N, int K, int part, cudaStream_t stream) {
  LIA_CHECK_ARG(n > 0 && n <= MAX_RANGES, "latent_expand: %d row ranges", n);
  ExpandArgs p{};
  p.n = n, p.K = K, p.part = part, p.col_tiles = N / COLS, p.C = C, p.ldc = ldc;
  long long all = 0;
  int out = 0;
  for (int i = 0; i < n; ++i) {
    LIA_CHECK_ARG(first[i] + rows[i] < (1ll << 31), "latent_expand: the cache has too many rows");
    p.row0[i] = (int)first[i], p.rows[i] = rows[i], p.tile0[i] = p.tiles, p.out0[i] = out;
    p.tiles += (rows[i] + ROWS - 1) / ROWS;
    out += rows[i];
    all = std::max(all, first[i] + rows[i]);
  }
  CUtensorMap rows_map, w_map;
  int rc = lia_make_tmap_2d(&rows_map, cache, (uint64_t)all, (uint64_t)K, (uint64_t)D, ROWS);
  if (rc == LIA_OK) rc = lia_make_tmap_2d(&w_map, W, (uint64_t)N, (uint64_t)K, (uint64_t)K, COLS);
  if (rc != LIA_OK) return rc;
  const int smem = smem_of(K), groups = std::max(1, std::min(p.col_tiles, lia_sm_count() / p.tiles));
  LIA_CUDA(cudaFuncSetAttribute(latent_expand_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_of(MAX_K)));
  int* timeouts = lia_timeout_word();
  LIA_CHECK_ARG(timeouts != nullptr, "lia_latent_attn_expanded: no host memory for the count of timeouts");
  lia_launch(latent_expand_kernel, dim3(p.tiles * groups), dim3(THREADS), smem, stream, rows_map, w_map, p, timeouts);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}
