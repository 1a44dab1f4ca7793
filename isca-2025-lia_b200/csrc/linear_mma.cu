// C[b][m][n] = scale * sum_k A[b][m][k] * W[b][n][k] on the tensor cores for the projections that the tcgen05 GEMM does not take: fp32
// inputs, fp32 results, batches of small matrices (a query carried into the latent space and back, keys and values expanded from latents, the
// gates of a block-diagonal recurrent unit, logits, models in fp32).
//
// fp32 operands enter as three bf16 parts (mma.cuh): an fp32 x bf16 product is three bf16 products, fp32 x fp32 six (of the nine, those whose
// factors together lie less than 24 bits below the highest).  Sums of 32 channels are made apart, the high products in one chain and the rest
// in another, and added to the running ones in fp32, because the tensor cores cut sums off instead of rounding them.  An infinity has no parts (its
// products with the other factor's parts, 0 or of the other sign, are NaN), so a sum that is not finite is formed again in one FMA chain.
//
// Bound: tensor cores (mma.sync m16n8k16).  128 x (16 NT) tile per block of 8 warps (4 x 2), a warp owns 32 x 8 NT; 32 channels per stage, two
// stages; bf16 operands come by cp.async, fp32 ones through registers, where they are split.
#include <type_traits>

#include "mma.cuh"

namespace {

constexpr int TM = 128, TKC = 32;          // rows per block, channels per stage

// rows of 4 chunks of 16 bytes: the chunk's place is turned by the row pair, so that 8 rows of one chunk touch all banks
__device__ __forceinline__ uint32_t at4(uint32_t base, int r, int c) { return base + (uint32_t)(r * 4 + (c ^ ((r >> 1) & 3))) * 16u; }

// One operand's tile of R rows: NP = 1 -- bf16 by cp.async; NP = 3 -- fp32 into registers (fetch), split and stored later (put).
template <int NP, int R> struct Tile {
  static constexpr int BYTES = NP * R * TKC * 2;
  static constexpr int IT = R * 4 / 256;   // 16-byte bf16 chunks (8 channels) per thread
  float4 v[NP == 3 ? IT : 1][2];

  __device__ __forceinline__ void fetch(const void* src, long long ld, int row0, int rows, int k0, int K, uint32_t dst) {
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      const int e = threadIdx.x + i * 256, r = e >> 2, c = e & 3, k = k0 + c * 8;
      const bool in = row0 + r < rows && k < K;
      if constexpr (NP == 1) {
        const bf16* p = reinterpret_cast<const bf16*>(src) + (in ? (size_t)(row0 + r) * ld + k : 0);
        cp_async16(at4(dst, r, c), p, in ? 16 : 0);
      } else {
        v[i][0] = v[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) {
          const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + (size_t)(row0 + r) * ld + k);
          v[i][0] = p[0];
          v[i][1] = p[1];
        }
      }
    }
  }
  __device__ __forceinline__ void put(uint32_t dst) {
    if constexpr (NP == 3) {
#pragma unroll
      for (int i = 0; i < IT; ++i) {
        const int e = threadIdx.x + i * 256, r = e >> 2, c = e & 3;
        uint32_t p[3][4];
        split3(v[i][0].x, v[i][0].y, p[0][0], p[1][0], p[2][0]);
        split3(v[i][0].z, v[i][0].w, p[0][1], p[1][1], p[2][1]);
        split3(v[i][1].x, v[i][1].y, p[0][2], p[1][2], p[2][2]);
        split3(v[i][1].z, v[i][1].w, p[0][3], p[1][3], p[2][3]);
#pragma unroll
        for (int s = 0; s < 3; ++s)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at4(dst + s * R * TKC * 2, r, c)), "r"(p[s][0]), "r"(p[s][1]), "r"(p[s][2]), "r"(p[s][3]) : "memory");
      }
    }
  }
};

// Row ranges of several sources as one problem (OUT_PARTS): range i has rows[i] rows at src[i], results from row out0[i] on, tiles from tile0[i] on
struct RowRanges {
  static constexpr int MAX = 16;
  int n, tile0[MAX], rows[MAX], out0[MAX];
  const bf16* src[MAX];
};
struct NoRanges {};

enum { OUT_F32, OUT_BF16, OUT_PARTS };     // OUT_PARTS: column n = group * part + c goes, as three bf16 parts, to [m][group][3][part]

// sum_k a[k] w[k] in one chain, as far as it is not settled
template <int NA, int NW> __device__ __noinline__ float plain_dot(const void* a, size_t a_at, const void* w, size_t w_at, int K) {
  float s = 0.f;
  for (int k = 0; k < K && s == s; ++k) {
    const float x = NA == 3 ? reinterpret_cast<const float*>(a)[a_at + k] : __bfloat162float(reinterpret_cast<const bf16*>(a)[a_at + k]);
    const float y = NW == 3 ? reinterpret_cast<const float*>(w)[w_at + k] : __bfloat162float(reinterpret_cast<const bf16*>(w)[w_at + k]);
    s = fmaf(x, y, s);
  }
  return s;
}

template <int NA, int NW, int NT, int OUT>
__global__ void __launch_bounds__(256) linear_mma_kernel(const void* __restrict__ A, long long lda, long long sA, const void* __restrict__ Wt, long long ldw,
                                                         long long sW, void* __restrict__ C, long long ldc, long long sC, int M, int N, int K, float scale,
                                                         int part, const std::conditional_t<OUT == OUT_PARTS, RowRanges, NoRanges> ranges) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int TN = 16 * NT, AB = Tile<NA, TM>::BYTES, WB = Tile<NW, TN>::BYTES;
  constexpr bool SPLIT = NA * NW > 1;
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t sm = smem_u32(smem);
  const int b = blockIdx.z, n0 = blockIdx.x * TN;
  int m0 = blockIdx.y * TM;
  if constexpr (OUT == OUT_PARTS) {
    int i = 0;
    while (i + 1 < ranges.n && (int)blockIdx.y >= ranges.tile0[i + 1]) ++i;
    m0 = ((int)blockIdx.y - ranges.tile0[i]) * TM;
    M = ranges.rows[i];
    A = ranges.src[i];
    C = reinterpret_cast<bf16*>(C) + (size_t)ranges.out0[i] * ldc;
  }
  A = reinterpret_cast<const char*>(A) + (size_t)b * sA * (NA == 3 ? 4 : 2);
  Wt = reinterpret_cast<const char*>(Wt) + (size_t)b * sW * (NW == 3 ? 4 : 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 8 * NT;

  float acc[2][NT][4], hi[2][NT][4], rest[SPLIT ? 2 : 1][SPLIT ? NT : 1][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[i][n][e] = hi[i][n][e] = 0.f;
        if constexpr (SPLIT) rest[i][n][e] = 0.f;
      }

  Tile<NA, TM> ta;
  Tile<NW, TN> tw;
  const int stages = (K + TKC - 1) / TKC;
  ta.fetch(A, lda, m0, M, 0, K, sm);
  tw.fetch(Wt, ldw, n0, N, 0, K, sm + AB);
  cp_async_commit();
  ta.put(sm);
  tw.put(sm + AB);
  for (int s = 0; s < stages; ++s) {
    const uint32_t as = sm + (s & 1) * (AB + WB), ws = as + AB, an = sm + ((s + 1) & 1) * (AB + WB);
    cp_async_wait<0>();
    __syncthreads();                         // stage s is there, and everybody is done with stage s - 1
    if (s + 1 < stages) {
      ta.fetch(A, lda, m0, M, (s + 1) * TKC, K, an);
      tw.fetch(Wt, ldw, n0, N, (s + 1) * TKC, K, an + AB);
      cp_async_commit();
    }
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      uint32_t a[2][NA][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int p = 0; p < NA; ++p) ldsm_x4(at4(as + p * TM * TKC * 2, wm + i * 16 + (lane & 15), 2 * kk + (lane >> 4)), a[i][p]);
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
#pragma unroll
        for (int q = NW - 1; q >= 0; --q) {
          uint32_t w[4];
          ldsm_x4(at4(ws + q * TN * TKC * 2, wn + n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * kk + ((lane >> 3) & 1)), w);
#pragma unroll
          for (int p = NA - 1; p >= 0; --p) {
            if (p + q > 2) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              if constexpr (SPLIT) {
                mma_bf16(p + q ? rest[i][n] : hi[i][n], a[i][p], w[0], w[1]);
                mma_bf16(p + q ? rest[i][n + 1] : hi[i][n + 1], a[i][p], w[2], w[3]);
              } else {
                mma_bf16(hi[i][n], a[i][p], w[0], w[1]);
                mma_bf16(hi[i][n + 1], a[i][p], w[2], w[3]);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if constexpr (SPLIT) {
            acc[i][n][e] += hi[i][n][e] + rest[i][n][e];
            rest[i][n][e] = 0.f;
          } else {
            acc[i][n][e] += hi[i][n][e];
          }
          hi[i][n][e] = 0.f;
        }
    if (s + 1 < stages) {
      ta.put(an);
      tw.put(an + AB);
    }
  }

#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int m = m0 + wm + i * 16 + g + u * 8;
      if (m >= M) continue;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int col = n0 + wn + n * 8 + 2 * t;
        if (col >= N) continue;
        if constexpr (SPLIT) {
          if (!(fabsf(acc[i][n][2 * u]) < INFINITY)) acc[i][n][2 * u] = plain_dot<NA, NW>(A, (size_t)m * lda, Wt, (size_t)col * ldw, K);
          if (col + 1 < N && !(fabsf(acc[i][n][2 * u + 1]) < INFINITY)) acc[i][n][2 * u + 1] = plain_dot<NA, NW>(A, (size_t)m * lda, Wt, (size_t)(col + 1) * ldw, K);
        }
        const float x = acc[i][n][2 * u] * scale, y = acc[i][n][2 * u + 1] * scale;
        if constexpr (OUT == OUT_F32) {
          float* p = reinterpret_cast<float*>(C) + (size_t)b * sC + (size_t)m * ldc + col;
          if (col + 1 < N && reinterpret_cast<uintptr_t>(p) % 8 == 0) {
            *reinterpret_cast<float2*>(p) = make_float2(x, y);
          } else {
            p[0] = x;
            if (col + 1 < N) p[1] = y;
          }
        } else if constexpr (OUT == OUT_BF16) {
          bf16* p = reinterpret_cast<bf16*>(C) + (size_t)b * sC + (size_t)m * ldc + col;
          if (col + 1 < N && reinterpret_cast<uintptr_t>(p) % 4 == 0) {
            *reinterpret_cast<uint32_t*>(p) = pack_bf16x2(x, y);
          } else {
            p[0] = __float2bfloat16_rn(x);
            if (col + 1 < N) p[1] = __float2bfloat16_rn(y);
          }
        } else {
          const int grp = col / part, c = col - grp * part;
          uint32_t h, md, lo;
          split3(x, y, h, md, lo);
          uint32_t* p = reinterpret_cast<uint32_t*>(reinterpret_cast<bf16*>(C) + (size_t)m * ldc + (size_t)grp * 3 * part + c);
          p[0] = h;
          p[part / 2] = md;
          p[part] = lo;
        }
      }
    }
}

template <int NA, int NW, int NT, int OUT>
int run(const void* A, long long lda, long long sA, const void* W, long long ldw, long long sW, void* C, long long ldc, long long sC, int M, int N, int K,
        int batch, float scale, cudaStream_t stream) {
  constexpr int smem = 2 * (Tile<NA, TM>::BYTES + Tile<NW, 16 * NT>::BYTES);
  if (smem > 48 * 1024) LIA_CUDA(cudaFuncSetAttribute(linear_mma_kernel<NA, NW, NT, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const dim3 grid((N + 16 * NT - 1) / (16 * NT), (M + TM - 1) / TM, batch);
  lia_launch(linear_mma_kernel<NA, NW, NT, OUT>, dim3(grid), dim3(256), smem, stream, A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, scale, 0, NoRanges{});
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

}  // namespace

bool linear_mma_takes(const void* A, int a_f32, long long lda, long long sA, const void* W, int w_f32, long long ldw, long long sW, int M, int K, int batch) {
  const int na = a_f32 ? 4 : 8, nw = w_f32 ? 4 : 8;
  return (a_f32 || !w_f32) && K % 8 == 0 && lda % na == 0 && sA % na == 0 && ldw % nw == 0 && sW % nw == 0 &&
         (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0 && (M + TM - 1) / TM <= 65535 && batch <= 65535;
}

int linear_mma(const void* A, int a_f32, long long lda, long long sA, const void* W, int w_f32, long long ldw, long long sW, void* C, int c_f32, long long ldc,
               long long sC, int M, int N, int K, int batch, float scale, cudaStream_t stream) {
  if (a_f32 && w_f32) {
    if (c_f32) return run<3, 3, 4, OUT_F32>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
    return run<3, 3, 4, OUT_BF16>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
  }
  if (a_f32) {
    if (c_f32) return run<3, 1, 4, OUT_F32>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
    return run<3, 1, 4, OUT_BF16>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
  }
  if (c_f32) return run<1, 1, 8, OUT_F32>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
  return run<1, 1, 8, OUT_BF16>(A, lda, sA, W, ldw, sW, C, ldc, sC, M, N, K, batch, scale, stream);
}

// bf16 x bf16 for up to 16 row ranges, the results one range after the other as three bf16 parts, `part` columns (a multiple of 2) at a
// time: C [rows][N / part][3][part], rows ldc numbers apart
int linear_mma_parts(const bf16* const* src, const int* rows, int n, long long lda, const bf16* W, bf16* C, long long ldc, int N, int K, int part, cudaStream_t stream) {
  LIA_CHECK_ARG(n > 0 && n <= RowRanges::MAX, "linear_mma_parts: %d row ranges", n);
  RowRanges r{};
  r.n = n;
  int tiles = 0, out = 0;
  for (int i = 0; i < n; ++i) {
    r.src[i] = src[i];
    r.rows[i] = rows[i];
    r.tile0[i] = tiles;
    r.out0[i] = out;
    tiles += (rows[i] + TM - 1) / TM;
    out += rows[i];
  }
  LIA_CHECK_ARG(tiles <= 65535, "linear_mma_parts: too many rows (%d)", out);
  constexpr int NT = 8, smem = 2 * (Tile<1, TM>::BYTES + Tile<1, 16 * NT>::BYTES);
  lia_launch(linear_mma_kernel<1, 1, NT, OUT_PARTS>, dim3(dim3((N + 16 * NT - 1) / (16 * NT), tiles, 1)), dim3(256), smem, stream, nullptr, lda, 0, W, K, 0, C, ldc, 0, 0, N, K,
                                                                                                              1.0f, part, r);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}
