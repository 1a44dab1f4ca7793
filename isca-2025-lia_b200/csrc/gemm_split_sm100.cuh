// Projections of 129 and more rows whose tiles leave SMs idle: the CTAs of a cluster take the parts of one tile's K, and the parts meet in shared memory.
//
// A CTA that runs the whole of K is bound by what one SM draws from L2 (96 KB a microsecond, 48 KB per 64 of K for a tile of 128 x 256), so 231 x 2560 x 10240 took 38 us on 80 SMs with
// HBM and tensor cores idle; in three parts on 120 SMs it takes 22.  At the end each CTA brings its fp32 sums from TMEM to its shared memory (the ring of stages is free by then) and sends every
// other CTA of the cluster that one's slice of the rows by one bulk copy (stores to the other CTAs' shared memory by 16 bytes a thread: 9 KB a microsecond, 24 us in all); there they are added in
// the order of K and go through the epilogue of gemm_shared.cuh.  A tile's sums depend on the number of parts alone, never on timing.
// Waits are bounded: a CTA that gives up sends NaN, and a word in host memory counts it (lia_moe_timeouts_seen()).
#pragma once
#include "gemm_shared.cuh"

int* lia_timeout_word();                                           // moe_sm100.cu

namespace {

// the sums that replace the ring: this CTA's, and the others' of its slice of rows
__host__ __device__ constexpr int split_bytes(int bn, int split) { return (2 * split - 1) * ((TILE_A + split - 1) / split) * bn * 4; }

template <int BN, int STAGES> struct SplitShape {
  static constexpr int STAGE_BYTES = (TILE_A + BN) * BLOCK_K * 2;
  static constexpr int MOST = BN == 256 ? 4 : 8;                   // CTAs that share a tile
  static constexpr int BARS = STAGES * STAGE_BYTES > split_bytes(BN, MOST) ? STAGES * STAGE_BYTES : split_bytes(BN, MOST);
  static constexpr int SMEM = BARS + (2 * STAGES + 2) * 8 + 16 + 1024;
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ EpiParams p,
                                                                     int k_blocks, int tiles_a, int split, int* timeouts) {
  using L = SplitShape<BN, STAGES>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u, bars = base + L::BARS;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  const uint32_t done_bar = bars + 8u * (2 * STAGES), recv_bar = done_bar + 8u;
  volatile uint32_t* tmem_ptr = reinterpret_cast<volatile uint32_t*>(gen + L::BARS + (2 * STAGES + 2) * 8);
  volatile int* dead = reinterpret_cast<volatile int*>(const_cast<uint32_t*>(tmem_ptr + 1));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_ctarank(), tile = blockIdx.x / split, ta = tile % tiles_a, tb = tile / tiles_a;
  const int kb0 = k_blocks * rank / split, kb1 = k_blocks * (rank + 1) / split;

  if (tid == 0) {
    *dead = 0;
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB) : "memory");
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    mbar_init(recv_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_ptr)), "r"((uint32_t)BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = *tmem_ptr;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0 && lane == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!wait_for(empty_bar(stage), phase ^ 1u, dead)) break;
      mbar_expect_tx(full_bar(stage), L::STAGE_BYTES);
      tma_load_2d(base + stage * L::STAGE_BYTES, &tmA, kb * BLOCK_K, ta * TILE_A, full_bar(stage));
      tma_load_2d(base + stage * L::STAGE_BYTES + TILE_A * BLOCK_K * 2, &tmB, kb * BLOCK_K, tb * BN, full_bar(stage));
      if (++stage == STAGES) stage = 0, phase ^= 1u;
    }
  } else if (warp == 1 && lane == 0) {
    constexpr uint32_t idesc = make_idesc(TILE_A, BN);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!wait_for(full_bar(stage), phase, dead)) break;
      tcgen05_fence_after();
      const uint64_t da = make_smem_desc(base + stage * L::STAGE_BYTES), db = make_smem_desc(base + stage * L::STAGE_BYTES + TILE_A * BLOCK_K * 2);
#pragma unroll
      for (int k = 0; k < BLOCK_K / UMMA_K; ++k) tcgen05_mma_f16(tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
      tcgen05_commit(empty_bar(stage));
      if (++stage == STAGES) stage = 0, phase ^= 1u;
    }
    tcgen05_commit(done_bar);
  }
  __syncwarp();

  // a thread finishes the columns 8 piece .. 8 piece + 7 of every PASS-th row of this CTA's slice
  constexpr int PIECES = BN / 8, PASS = NUM_THREADS / PIECES, MOST = (TILE_A / 2 + PASS - 1) / PASS;
  const int slice = (TILE_A + split - 1) / split, piece = tid % PIECES, i0 = tid / PIECES, n = tb * BN + piece * 8;
  const int m0 = ta * TILE_A + rank * slice, rows = min(min(slice, TILE_A - rank * slice), p.M - m0);
  float bias[8];
  uint4 res[MOST];
  if (n < p.N) {
    epilogue_load_bias8(p, n, bias);
#pragma unroll
    for (int k = 0; k < MOST; ++k) res[k] = i0 + k * PASS < rows ? epilogue_load_residual8(p, m0 + i0 + k * PASS, n) : make_uint4(0, 0, 0, 0);
  }
  const bool alive = warp_wait(done_bar, 0u, dead);
  tcgen05_fence_after();
  if (!alive) {                                                    // loads in flight end before anything is written over the ring
    volatile int none = 0;
    if (tid == 0) {
      atomicAdd_system(timeouts, 1);
      for (int s = 0; s < STAGES && s < kb1 - kb0; ++s) wait_for(full_bar(s), 0u, &none);
    }
  }
  const uint32_t theirs = base + (uint32_t)(split * slice * BN) * 4u;
  if (tid == 0 && rows > 0) mbar_expect_tx(recv_bar, (uint32_t)((split - 1) * rows * BN) * 4u);
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");                   // this CTA's stages are read no more
  {
    const int row = (warp & 3) * 32 + lane;
#pragma unroll 1
    for (int c0 = (warp >> 2) * (BN / 2); c0 < ((warp >> 2) + 1) * (BN / 2); c0 += 32) {
      uint32_t v[32];
      tmem_ld32(tmem + c0 + ((uint32_t)((warp & 3) * 32) << 16), v);
      tmem_ld_wait();
      if (!alive) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0x7fc00000u;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)                                  // a piece's place is turned by its row: 8 lanes touch all banks
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(base + (uint32_t)(row * BN) * 4u + (uint32_t)(((c0 >> 2) + j) ^ (row & 7)) * 16u), "r"(v[4 * j]),
                     "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3]) : "memory");
    }
  }
  fence_proxy_async_smem();
  tcgen05_fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (tid == 0) {
    for (int d = 1; d < split; ++d) {
      const int to = rank + d < split ? rank + d : rank + d - split, first = to * slice, n_rows = min(min(slice, TILE_A - first), p.M - ta * TILE_A - first);
      if (n_rows > 0)
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         mapa_u32(theirs + (uint32_t)((rank < to ? rank : rank - 1) * slice * BN) * 4u, to)),
                     "r"(base + (uint32_t)(first * BN) * 4u), "r"((uint32_t)(n_rows * BN) * 4u), "r"(mapa_u32(recv_bar, to))
                     : "memory");
    }
  }
  const bool arrived = rows <= 0 || warp_wait(recv_bar, 0u, dead);
  if (!arrived && lane == 0 && warp == 0) atomicAdd_system(timeouts, 1);
  if (n < p.N) {
#pragma unroll
    for (int k = 0; k < MOST; ++k) {
      const int i = i0 + k * PASS, row = rank * slice + i;
      if (i >= rows) break;
      float f[8] = {};
      for (int s = 0; s < split; ++s) {
        const uint32_t src = s == rank ? base + (uint32_t)(row * BN) * 4u : theirs + (uint32_t)(((s < rank ? s : s - 1) * slice + i) * BN) * 4u;
        float u[8];
#pragma unroll
        for (int half = 0; half < 2; ++half)
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(u[4 * half]), "=f"(u[4 * half + 1]), "=f"(u[4 * half + 2]), "=f"(u[4 * half + 3])
                       : "r"(src + (uint32_t)((2 * piece + half) ^ (row & 7)) * 16u));
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = s ? f[e] + u[e] : u[e];
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = arrived ? bf16r(f[e]) : NAN;
      epilogue_finish8(p, m0 + i, n, f, bias, res[k]);
    }
  }
  cluster_sync_all();                                              // the copies out of this CTA's shared memory have ended
  __syncthreads();
  if (warp == 2) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
  }
}

template <int BN, int STAGES> int launch_split(const Plan& pl, const CUtensorMap& tmA, const CUtensorMap& tmB, const EpiParams& ep, cudaStream_t stream) {
  using L = SplitShape<BN, STAGES>;
  static_assert(L::SMEM <= 232448, "shared memory budget exceeded");
  auto kern = gemm_split_kernel<BN, STAGES>;
  LIA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM));
  int* timeouts = lia_timeout_word();
  LIA_CHECK_ARG(timeouts != nullptr, "lia_gemm_bf16: no host memory for the count of timeouts");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = lia_pdl_enabled() ? 2 : 1;
  LIA_CUDA(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, ep, pl.k_blocks, pl.tiles_a, pl.split, timeouts));
  return LIA_OK;
}

}  // namespace
