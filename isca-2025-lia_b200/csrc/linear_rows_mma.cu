// C[b][m][n] = sum_k A[b][m][k] W[b][n][k] on mma.sync for bf16 numbers where few rows or few columns leave the tcgen05 GEMM's tiles empty: the projections of decoded tokens,
// logits, gates and routers.
//
// A step of decoded tokens is a chain of small projections, and what the tcgen05 GEMM takes for one is latency: tensor maps, barriers, TMEM, a ring that fills, partial sums that change
// hands.  Here the weights go straight from global memory into the operands' registers: 16 bytes of a weight row are two operands' worth of k, and as the rows of A are read the same
// way the order of the k within 32 does not matter.  Where the caller says that no work in flight on the stream writes them (`resident`: a model's weights) they are asked for before the
// previous kernel has ended.  (Non-coherent loads; by ld.global.cg an engine session of four requests takes 3335 us in place of 3220.)  A block makes 16 or 32 columns of 8 to 32 rows, its 8 warps an eighth of K
// each; they meet once, in shared memory.
//
// The tensor cores cut sums off below the 24th bit: those over 32 k are made apart and added in fp32.  Where the result is fp32 those over 16 are, what a warp's sum rounds off is added up apart
// and the warps' sums meet in 64 bits; against 64 bits: K = 128, 1024, 4096: off by 4.3e-8, 4.4e-8, 4.4e-8 (FMA chains: 4.8e-8, 6.9e-8, 9.5e-8).  A row's result does not depend on the rows beside
// it: neither the share of a warp nor the order of its sums looks at M.
//
// Bound: latency, then the rows' way from L2 (every block reads its rows of A whole).
#include <math.h>

#include <type_traits>

#include "linear_rows_mma.cuh"
#include "mma.cuh"

namespace {

constexpr int WARPS = 8;

struct RowsArgs {
  const bf16 *A, *W;
  void* C;
  long long lda, sA, ldw, sW, ldc, sC;
  int M, N, K;
  float scale;
  const float* bias;                           // gates
  int mode;
  float cap;
  int resident;
};

enum { OUT_GEMM, OUT_FP32, OUT_ROUNDED, OUT_GATES };              // GEMM: bf16, whole vectors, nothing kept of what the sums round off

// A block: 8 NT rows times 16 MT columns.  CB: blocks of 32 k in registers at a time
template <int NT, int MT, int CB> struct Form {
  static constexpr int ROWS = 8 * NT, COLS = 16 * MT, PITCH = COLS + 4, SMEM = WARPS * ROWS * PITCH * 4;
  static constexpr int REGS = 4 * NT * MT + CB * 4 * (2 * MT + NT);                  // of the sums and operands
};
template <int NT, int MT, int CB, int OUT>
__global__ void __launch_bounds__(WARPS * 32, Form<NT, MT, CB>::REGS + (OUT == OUT_GEMM ? 0 : 4 * NT * MT) <= 112 ? 2 : 1) linear_rows_kernel(const RowsArgs p) {
  using F = Form<NT, MT, CB>;
  extern __shared__ __align__(16) float red[];                     // [WARPS][ROWS][PITCH]
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * F::COLS, m0 = blockIdx.z * F::ROWS, blocks = (p.K + 31) >> 5;
  const int first = (int)((long long)blocks * warp / WARPS), last = (int)((long long)blocks * (warp + 1) / WARPS);
  const bf16* A = p.A + (size_t)blockIdx.y * p.sA + t * 8;
  const bf16* W = p.W + (size_t)blockIdx.y * p.sW + t * 8;
  uint4 w[CB][MT][2], x[CB][NT];
  auto weights = [&](int b0) {
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int k = (b0 + b) * 32;
      const bool live = b0 + b < last && k + t * 8 < p.K;
#pragma unroll
      for (int i = 0; i < 2 * MT; ++i) w[b][i >> 1][i & 1] = live ? ldg_stream(W + (size_t)min(n0 + g + 8 * i, p.N - 1) * p.ldw + k) : make_uint4(0, 0, 0, 0);
    }
  };
  if (!p.resident) pdl_wait();
  weights(first);
  pdl_wait();
  float acc[NT][MT][4] = {}, left[OUT == OUT_GEMM ? 1 : NT][MT][4] = {};
  auto add = [&](const float* c, int nt, int mt) {                 // what the sum rounds off is kept, exactly (Knuth's two-sum), in a sum of its own
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float& sum = acc[nt][mt][e];
      const float next = sum + c[e], back = next - sum;
      left[OUT == OUT_GEMM ? 0 : nt][mt][e] += (sum - (next - back)) + (c[e] - back);
      sum = next;
    }
  };
#pragma unroll 1
  for (int b0 = first; b0 < last; b0 += CB) {
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int k = (b0 + b) * 32;
      const bool live = b0 + b < last && k + t * 8 < p.K;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) x[b][nt] = live ? ldg_act(A + (size_t)min(m0 + nt * 8 + g, p.M - 1) * p.lda + k) : make_uint4(0, 0, 0, 0);
    }
    if (b0 > first) weights(b0);
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      if (b0 + b >= last) break;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const uint4 u = w[b][mt][0], d = w[b][mt][1];
        const uint32_t lo[4] = {u.x, d.x, u.y, d.y}, hi[4] = {u.z, d.z, u.w, d.w};
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float c[4];
          mma_bf16_first(c, lo, x[b][nt].x, x[b][nt].y);
          if constexpr (OUT == OUT_GEMM) {
            mma_bf16(c, hi, x[b][nt].z, x[b][nt].w);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][mt][e] += c[e];
          } else {
            float c2[4];
            mma_bf16_first(c2, hi, x[b][nt].z, x[b][nt].w);
            add(c, nt, mt);
            add(c2, nt, mt);
          }
        }
      }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int e = 0; e < 4; ++e) red[(warp * F::ROWS + nt * 8 + 2 * t + (e & 1)) * F::PITCH + mt * 16 + g + 8 * (e >> 1)] =
            OUT == OUT_GEMM || !(fabsf(acc[nt][mt][e]) < INFINITY) ? acc[nt][mt][e] : acc[nt][mt][e] + left[OUT == OUT_GEMM ? 0 : nt][mt][e];     // (of an infinity nothing is left)
  __syncthreads();
  for (int i = threadIdx.x; i < F::ROWS * 2 * MT; i += WARPS * 32) {           // 8 columns of a row
    const int r = i / (2 * MT), m = m0 + r, c0 = i % (2 * MT) * 8, n = n0 + c0;
    if (m >= p.M || n >= p.N) continue;
    using Sum = typename std::conditional<OUT == OUT_GEMM, float, double>::type;
    Sum sum[8] = {};
#pragma unroll
    for (int k = 0; k < WARPS; ++k) {
      const float4* s = reinterpret_cast<const float4*>(red + (k * F::ROWS + r) * F::PITCH + c0);
      const float4 a = s[0], b = s[1];
      sum[0] += a.x, sum[1] += a.y, sum[2] += a.z, sum[3] += a.w, sum[4] += b.x, sum[5] += b.y, sum[6] += b.z, sum[7] += b.w;
    }
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = (float)sum[e];
    if constexpr (OUT == OUT_GEMM) {
      *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.C) + (size_t)m * p.ldc + n) = pack8(v);        // (N and ldc are multiples of 8)
    } else {
      const int live = min(8, p.N - n);
      const size_t at = (size_t)blockIdx.y * p.sC + (size_t)m * p.ldc + n;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < live) {
          if constexpr (OUT == OUT_FP32) {
            reinterpret_cast<float*>(p.C)[at + e] = v[e] * p.scale;
          } else if constexpr (OUT == OUT_ROUNDED) {
            reinterpret_cast<bf16*>(p.C)[at + e] = __float2bfloat16_rn(v[e] * p.scale);
          } else {
            float z = v[e] + (p.bias ? p.bias[n + e] : 0.f);
            if (p.mode == 1) {
              z = p.cap * tanhf(z / p.cap);
              if (n + e >= p.N / 2) z = fminf(z, 0.f) - log1pf(expf(-fabsf(z)));
            } else if (p.mode == 2) {
              z = 1.0f / (1.0f + expf(-z));
            }
            reinterpret_cast<float*>(p.C)[at + e] = z;
          }
        }
    }
  }
}

template <int NT, int MT, int CB, int OUT> int launch_rows_as(const RowsArgs& p, int batch, cudaStream_t stream) {
  using F = Form<NT, MT, CB>;
  if (F::SMEM > 48 * 1024) LIA_CUDA(cudaFuncSetAttribute(linear_rows_kernel<NT, MT, CB, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, F::SMEM));
  lia_launch(linear_rows_kernel<NT, MT, CB, OUT>, dim3((p.N + F::COLS - 1) / F::COLS, batch, (p.M + F::ROWS - 1) / F::ROWS), dim3(WARPS * 32), F::SMEM, stream, p);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}
// Few rows a block, and all of a warp's share of K at once, as long as every block has an SM; then more rows, two blocks an SM, and more columns, which read the rows less often.  No form
// changes a number.  Gates of 16 x 2048, 8 | 200 | 2048 | 4096 rows: blocks of 8 rows 4.0 | 4.4 | 8.8 us, of 16 4.7 | 5.4 | 5.7 | 8.1 (with less at a time), of 32 7.5 | 8.3 | 8.8 | 8.9;
// 1024 x 2816 in bf16, 16 | 32 | 128 rows: 3.1 | 5.2, 3.1 | 3.5 | 9.5, 5.9 | 5.9 | 7.8; 2048 x 2048, 128 rows, 16 columns a block 11.5, 32 9.0.  Blocks of 24 rows where no more of them are needed:
// 2048 x 5632, 48 rows 14.1 -> 11.8, 1024 x 8192, 40 rows 13.8 -> 12.2.
template <int OUT> int launch_rows(const RowsArgs& p, int batch, cudaStream_t stream) {
  const long long sms = lia_sm_count(), narrow = (long long)((p.N + 15) / 16) * batch, by8 = narrow * ((p.M + 7) / 8), by16 = narrow * ((p.M + 15) / 16), by32 = narrow * ((p.M + 31) / 32);
  constexpr bool fp32 = OUT != OUT_GEMM;                           // twice the sums' registers
  constexpr int SOME = fp32 ? 6 : 8;
  const bool deep = p.K > SOME * 32 * WARPS;
  if (by8 <= sms) return deep ? launch_rows_as<1, 1, 12, OUT>(p, batch, stream) : launch_rows_as<1, 1, SOME, OUT>(p, batch, stream);
  if (p.M <= 8) return launch_rows_as<1, 1, SOME, OUT>(p, batch, stream);
  if (by16 <= sms) {
    if constexpr (!fp32)
      if (deep) return launch_rows_as<2, 1, 12, OUT>(p, batch, stream);
    return launch_rows_as<2, 1, 8, OUT>(p, batch, stream);
  }
  if (p.M <= 16) return launch_rows_as<2, 1, 4, OUT>(p, batch, stream);
  if constexpr (fp32) {
    if (by16 <= 2 * sms) return launch_rows_as<2, 1, 4, OUT>(p, batch, stream);
    return launch_rows_as<4, 1, 2, OUT>(p, batch, stream);
  } else {
    const bool by24 = (p.M + 23) / 24 == (p.M + 31) / 32;
    if (by32 <= sms) return by24 ? launch_rows_as<3, 1, 6, OUT>(p, batch, stream) : launch_rows_as<4, 1, 6, OUT>(p, batch, stream);
    if (by32 <= 2 * sms) return by24 ? launch_rows_as<3, 1, 4, OUT>(p, batch, stream) : launch_rows_as<4, 1, 3, OUT>(p, batch, stream);
    return by24 ? launch_rows_as<3, 2, 2, OUT>(p, batch, stream) : launch_rows_as<4, 2, 2, OUT>(p, batch, stream);
  }
}

}  // namespace

// The line looks at the weights alone, for the other side's sums are other ones: where no number of rows up to 128 is the slower one here.  In a chain of projections over 300 MB of weights,
// 1 | 16 | 32 | 48 | 64 | 128 rows: 1024 x 1024 5.7 | 5.9 | 6.6 | 7.6 | 7.8 | 10.9 us on the other side and 1.7 | 2.1 | 2.1 | 2.6 | 3.0 | 4.0 here, 1024 x 8192 9.2 | 10.0 | 11.8 | 14.2 | 15.2 |
// 26.7 and 7.0 | 7.5 | 9.4 | 12.5 | 14.7 | 18.3, 2048 x 5632 8.3 | 9.0 | 11.0 | 13.4 | 14.4 | 25.8 and 5.7 | 7.7 | 11.2 | 11.8 | 14.4 | 21.2, 4096 x 2048 7.7 | 8.1 | 9.3 | 10.6 | 11.4 | 18.7 and
// 3.6 | 5.4 | 6.6 | 7.8 | 9.3 | 16.8; beyond: 512 x 16384 10.7 | 11.9 and 13.2 | 17.5, 3072 x 4096 8.2 | 8.5 | 11.2 | 13.1 | 14.3 and 5.3 | 8.9 | 11.7 | 13.5 | 16.8, 4096 x 3072, 96 rows, 18.7 and
// 22.7, and, with 32 rows in blocks of 32, 1024 x 8192 11.8 and 15.0 (so that deep ones are taken where those of 16 have an SM each: 1184 columns).
// (lia_gemm_bf16 is not among its callers: OPT's operations one by one give the bits of the program that chains them in one launch, decode_program_sm100.cu, with the GEMM's sums.)
bool gemm_rows_takes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 128) return false;
  if (N <= 1184) return K <= 8192;
  if (N <= 2368) return K <= 5632 && (long long)N * K <= 11 << 20;
  return N <= 4096 && (long long)N * K <= 8 << 20;
}

int gemm_rows(const void* A, const void* W, void* C, int M, int N, int K, cudaStream_t stream) {
  const RowsArgs p{reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(W), C, K, 0, K, 0, N, 0, M, N, K, 1.f, nullptr, 0, 0.f, 1};
  return launch_rows<OUT_GEMM>(p, 1, stream);
}

bool linear_rows_takes(const void* A, long long lda, long long sA, const void* W, long long ldw, long long sW, int M, int K) {
  return (M + 7) / 8 <= 65535 && K % 8 == 0 && lda % 8 == 0 && sA % 8 == 0 && ldw % 8 == 0 && sW % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0;
}

int linear_rows(const void* A, long long lda, long long sA, const void* W, long long ldw, long long sW, void* C, int c_f32, long long ldc, long long sC, int M, int N, int K,
                int batch, float scale, int resident, cudaStream_t stream) {
  const RowsArgs p{reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(W), C, lda, sA, ldw, sW, ldc, sC, M, N, K, scale, nullptr, 0, 0.f, resident};
  return c_f32 ? launch_rows<OUT_FP32>(p, batch, stream) : launch_rows<OUT_ROUNDED>(p, batch, stream);
}

int linear_rows_gates(const void* A, long long lda, const void* W, const float* bias, float* out, int M, int N, int K, int mode, float cap, int resident, cudaStream_t stream) {
  const RowsArgs p{reinterpret_cast<const bf16*>(A), reinterpret_cast<const bf16*>(W), out, lda, 0, K, 0, N, 0, M, N, K, 1.f, bias, mode, cap, resident};
  return launch_rows<OUT_GATES>(p, 1, stream);
}
