// The matrix-state recurrences of linear_scan.cu (fixed decay) and mlstm.cu over long portions: chunks of L tokens on the tensor cores.
//
// With D[t][s] the product of the decays between s and t (times s's write gate), A[t] that of the decays up to t and S the state before the chunk:
//     O = (D o Q K^T) V + A o (Q S)         S' = A[L-1] S + K^T (w o V),  w[s] = D[L-1][s]
// Token by token a head's state costs 2 dim vdim FMAs and a butterfly per token on the CUDA cores, one token after the other; here a chunk is four
// contractions.  The inputs are bf16; what is computed in fp32 stays as exact as fp32: D o Q K^T, S and w o V enter their contractions as three bf16
// parts (mma.cuh), tensor-core sums are kept to a few instructions and then added in fp32, the state itself stays in fp32 registers.  All weights are
// products of decays (never quotients or differences of logarithms), so nothing can overflow that the token loop would keep.
//
// Split: a CTA owns 32 columns of one head of one portion, walks its chunks in order and computes the head's Q K^T again (a quarter of the work at 128 dims;
// more columns per CTA would leave SMs idle at the usual 100 to 150 slices).  8 warps contract: the two (L = 64) or four (L = 32, where 256 dims leave no
// room for longer chunks) of a row block share its Q S by rows of the state and its score blocks, and hand their parts of the output over in shared memory;
// for the update each owns dim / 8 rows of the state.  4 warps put the last chunk's output together, keep the normaliser and make the next chunk's w o V,
// one the next chunk's gates.  Q, K and V arrive by cp.async a chunk ahead.
//
// The hi parts' products are summed per instruction (exact but for the last bits) and added in fp32; only the lower parts stay in the tensor cores' sums,
// which truncate.  Against 64 bits, means over 6 to 10 inputs: 16 heads of 128 x 128, 1024 tokens: outputs off by 8.5e-8 (token loop: 12e-8), the state by 8e-8 (19e-8), 64
// tokens: 7.8e-8 (8.0e-8) and 6.1e-8 (12e-8); gated, 4 heads of 256 x 512, 503 and 400 tokens: outputs' median 1.5e-7 (1.9e-7), state 1.15e-7 (1.2e-7), normaliser as there.
// A chunk of 64 takes about 3.3 us, one of 32 at 256 dims 3.6, one after the other (a sequence's chunks cannot run at once): cutting the additions to half did not
// change that; the chain ldmatrix, mma, add, the two barriers and the instructions themselves bound it (thirteen warps run three programs; see the loops' unrolling).
// A portion of 2048 tokens: 16 heads of 128 x 128 533 us by tokens, 102 here, 4 heads of 256 x 512 878 and 227.
#include <math.h>

#include "common.cuh"
#include "mma.cuh"

int mlstm_take_state(const float* ws, const int* segs, int nseg, float* nst, float* mst, int H, int dim, cudaStream_t stream);      // mlstm.cu
int mlstm_scan_tokens(const void* q, const void* k, const void* v, int ld, const float* gates, float* St, float* nst, float* mst, float* ws, const int* segs, int below,
                      int nseg, int H, int dim, int vdim, float q_scale, float den_eps, float* o, cudaStream_t stream);
int decay_scan_tokens(const void* q, const void* k, int ldqk, const void* v, int ldv, const float* decay, float* St, const int* segs, int below, int nseg, int H, int G,
                      int dim, int vdim, float* o, cudaStream_t stream);                                                          // linear_scan.cu

namespace {

constexpr int COLS = 32;                       // columns of the state per CTA
constexpr int MW = 8;                          // contracting warps
constexpr int VP = COLS + 8;                   // row pitches in bf16 (16 bytes past a multiple of 128: ldmatrix without bank conflicts)
constexpr int OP = COLS + 4;                   // and of the output parts in floats
// A portion of fewer tokens is left to the token loops, whichever portions come with it (a portion's rounding must not depend on its company).  One portion of 24 tokens:
// 13 us there and 10 here, of 32: 14 and 11, 8 of 33: 44 and 29; but 16 of one token: 6 and 47, for a CTA fills an SM and its chunk costs the same few
// us however little it holds.  A prompt of 256 among 31 single tokens: 90 us all by tokens, 90 all in chunks, 42 split.
constexpr int SHORT = 32;
// Below this many tokens with a fixed decay the token loop rounds so little that scores summed in two chains would leave the outputs off by 1.02 to 1.08 times its error:
// they are summed with their rounding errors, 0.93 to 0.98 times, by a kernel of their own (from here on two chains: 0.98 at 64 tokens, 0.92 at 100; the errors kept for
// all portions: 28 us more of 216 for 2048 tokens, both ways in one kernel: 5).
constexpr int FEW = 64;

struct ChunkArgs {
  const bf16 *q, *k, *v;
  int ldqk, ldv;
  const float *decay, *gates;                  // [H] | [rows][2H]
  float *St, *nst, *mst, *ws;                  // ws: where the new n and m wait (null: straight into the state)
  const int* segs;
  int H, G, vdim;
  float q_scale, den_eps;
  float* o;
};

template <int DIM, int L> struct ChunkSmem {
  static constexpr int QP = DIM + 8, WPR = MW / (L / 16);
  bf16 q[2][L][QP], k[2][L][QP], v[2][L][VP];
  bf16 vw[2][3][L][VP];                        // parts of w o V
  bf16 s[3][COLS][QP];                         // parts of the state before the chunk
  alignas(16) float part[2][WPR][L][OP];         // of the output
  float D[2][32][33];                          // mLSTM
  alignas(16) float a[2][L], w[2][L], em[2][L];
  float rs[2][WPR][L], nq[2][L];               // row sums of the scores; q . n
  alignas(16) float n[DIM];
  float pw[L + 1];                             // powers of a fixed decay
  float total[2];
  alignas(16) int bad[2][COLS];                            // first token whose v is not finite
};

// Where a contracting warp's rows of the state begin in Q S, in steps of 16.  A step takes a warp some 470 clocks at 256 dims, a block of scores and its values five times that (more than its
// instructions, 2 KS + 12 beside a step's 12, for a step's are less of a chain), and the warps of a row block that have fewer blocks of scores take more steps.  The chain of two portions of 1003 tokens,
// 4 heads of 256 x 512: 132 us with a block counted by its instructions and all warps in the scores' loop, 125 without those that have none there and a block for nine steps, 118 for five.  Where
// two warps share a row block, six steps of one of them are a longer chain of fp32 additions and put outputs off by 1.006 times as much: five at most.  As many steps for each warp as before -- as
// shared now, outputs off by, in 1e-7, means over 24 inputs: four warps (256 x 512, up to six steps) 120 tokens 2.407 -- 2.408, 503 2.480 -- 2.478, 1003 2.773 -- 2.772; two (128 x 128, up to five)
// 64 tokens 0.776 -- 0.776, 200 0.829 -- 0.828, 1024 1.027 -- 1.028.
template <int RB, int WPR, int KS> struct Shares {
  int from[RB][WPR + 1];
  constexpr Shares() : from{} {
    for (int rb = 0; rb < RB; ++rb) {
      int load[WPR] = {}, steps[WPR] = {};
      for (int blk = 0; blk <= rb; ++blk) load[blk % WPR] += 3 * KS + 12;
      for (int ks = 0; ks < KS; ++ks) {
        int least = -1;
        for (int i = 0; i < WPR; ++i)
          if ((WPR > 2 || steps[i] < 5) && (least < 0 || load[i] < load[least])) least = i;
        load[least] += 12, ++steps[least];
      }
      for (int i = 0; i < WPR; ++i) from[rb][i + 1] = from[rb][i] + steps[i];
    }
  }
};
// all of them as one number of five bits each (as an array in constant memory they cost a portion of one chunk 0.2 of its 7.1 us)
template <int RB, int WPR, int KS> constexpr unsigned long long packed_shares() {
  static_assert(RB * (WPR + 1) * 5 <= 64 && KS < 32, "shares do not fit");
  const Shares<RB, WPR, KS> shares;
  unsigned long long v = 0;
  for (int rb = RB - 1; rb >= 0; --rb)
    for (int i = WPR; i >= 0; --i) v = v << 5 | (unsigned)shares.from[rb][i];
  return v;
}
template <int RB, int WPR, int KS> struct PackedShares {
  static constexpr unsigned long long value = packed_shares<RB, WPR, KS>();
};
template <int RB, int WPR, int KS> __device__ __forceinline__ int share_from(int rb, int i) { return (int)(PackedShares<RB, WPR, KS>::value >> (5 * (rb * (WPR + 1) + i))) & 31; }

// MLSTM: gates per token with a running-maximum stabiliser and a normaliser; else one decay per head, and the portions of SHORT to FEW - 1 tokens (few) or those of FEW and more.
template <bool MLSTM, int DIM, int L, bool few = false>
__global__ void __launch_bounds__((MW + 4 + MLSTM) * 32, 1) chunk_scan_kernel(ChunkArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  constexpr int RB = L / 16, WPR = MW / RB, KS = DIM / 16, NB = (RB + WPR - 1) / WPR, NTU = DIM / 64;
  extern __shared__ __align__(16) unsigned char raw[];
  ChunkSmem<DIM, L>& sm = *reinterpret_cast<ChunkSmem<DIM, L>*>(raw);
  const int seg = blockIdx.z, h = blockIdx.y, colb = blockIdx.x * COLS;
  const int slot = p.segs[4 * seg], row0 = p.segs[4 * seg + 2], len = p.segs[4 * seg + 3];
  if (len < (MLSTM || few ? SHORT : FEW) || (few && len >= FEW)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int H = p.H, vdim = p.vdim;
  const bf16* qb = p.q + (size_t)row0 * p.ldqk + (size_t)(h / (H / p.G)) * DIM;
  const bf16* kb = p.k + (size_t)row0 * p.ldqk + (size_t)(h / (H / p.G)) * DIM;
  const bf16* vb = p.v + (size_t)row0 * p.ldv + (size_t)h * vdim + colb;
  const int chunks = (len + L - 1) / L;

  const int aux = tid - MW * 32;
  constexpr int QC = DIM / 8, PIECES = 2 * L * QC / (MW * 32);
  auto fetch_qk = [&](int c, int piece) {      // rows beyond the portion and columns beyond vdim are zero
    const int b = c & 1, e = tid + piece * MW * 32, r = e / (2 * QC), j = e % (2 * QC), tok = c * L + r;
    const bool live = tok < len;
    const bf16* src = (j < QC ? qb + j * 8 : kb + (j - QC) * 8) + (live ? (size_t)tok * p.ldqk : 0);
    cp_async16(smem_u32(j < QC ? &sm.q[b][r][j * 8] : &sm.k[b][r][(j - QC) * 8]), src, live ? 16 : 0);
  };
  auto fetch_v = [&](int c) {                  // the helping warps read V before the others do
    const int b = c & 1;
#pragma unroll
    for (int e = aux; e < L * COLS / 8; e += 128) {
      const int r = e / (COLS / 8), col = e % (COLS / 8) * 8, tok = c * L + r;
      const bool live = tok < len && colb + col < vdim;
      cp_async16(smem_u32(&sm.v[b][r][col]), live ? vb + (size_t)tok * p.ldv + col : p.v, live ? 16 : 0);
    }
    cp_async_commit();
  };
  // ---- the gate warp: everything about a chunk's gates; m is carried along (lane = token, L = 32)
  float m = 0.f, next_i = 0.f, next_f = 0.f;
  auto read_gates = [&](int c) {
    next_i = next_f = 0.f;
    if (c * L + lane < len) {
      const float* gp = p.gates + (size_t)(row0 + c * L + lane) * 2 * H + h;
      next_i = __ldg(gp);
      next_f = __ldg(gp + H);
    }
  };
  auto gates = [&](int c) {
    const int b = c & 1, n = min(L, len - c * L);
    const float ig = next_i, fg = next_f;
    read_gates(c + 1);
    float before = m, after = m;
    // (like the scores' loop by four: whole, these loops push each other's instructions out of the cache.  Two portions of 1003 tokens, 4 heads of 256 x 512, before the warps' shares were as
    // they are now: 139 us whole, 132 by four, 136 by two and one at a time)
#pragma unroll 4
    for (int t = 0; t < 32; ++t) {
      const float f = __shfl_sync(0xffffffffu, fg, t), i = __shfl_sync(0xffffffffu, ig, t);
      const float next = t < n ? fmaxf(f + m, i) : m;
      if (lane == t) before = m, after = next;
      m = next;
    }
    if (c > 0) asm volatile("bar.sync 2, 160;" ::: "memory");           // the chunk before the last has left this chunk's buffers
    const float a = lane < n ? expf(fg + before - after) : 1.f, w = lane < n ? expf(ig - after) : 0.f;
    float prod = 0.f, all = 1.f, mine = 1.f;
#pragma unroll 4
    for (int t = 0; t < 32; ++t) {
      const float at = __shfl_sync(0xffffffffu, a, t);
      all *= at;
      prod = lane < t ? prod * at : (lane == t ? w : 0.f);
      sm.D[b][t][lane] = prod;
      if (lane == t) mine = all;
    }
    sm.a[b][lane] = mine;
    sm.w[b][lane] = prod;
    sm.em[b][lane] = expf(-after);
    if (lane == 0) sm.total[b] = all;
    if (c > 0) asm volatile("bar.sync 3, 160;" ::: "memory");           // for weigh
  };
  // ---- the 4 helping warps: the chunk's w o V in three parts.  A v that is not finite must not reach earlier tokens through their zero scores: it leaves
  // the tile, and the column's outputs are NaN from its token on
  auto weigh = [&](int c) {
    const int b = c & 1, n = min(L, len - c * L);
#pragma unroll 4
    for (int e = aux; e < L * COLS / 2; e += 128) {
      const int s = e / (COLS / 2), col = (e - s * (COLS / 2)) * 2;
      uint32_t* src = reinterpret_cast<uint32_t*>(&sm.v[b][s][col]);
      float x, y;
      unpack_bf16x2(*src, x, y);
      const float w = MLSTM ? sm.w[b][s] : (s < n ? sm.pw[n - 1 - s] : 0.f);
      if (!(fabsf(x) < INFINITY && fabsf(y) < INFINITY)) {
        if (!(fabsf(x) < INFINITY)) atomicMin(&sm.bad[b][col], s);
        if (!(fabsf(y) < INFINITY)) atomicMin(&sm.bad[b][col + 1], s);
        *src = pack_bf16x2(fabsf(x) < INFINITY ? x : 0.f, fabsf(y) < INFINITY ? y : 0.f);
      }
      uint32_t hi, mid, lo;
      split3_finite(x * w, y * w, hi, mid, lo);
      *reinterpret_cast<uint32_t*>(&sm.vw[b][0][s][col]) = hi;
      *reinterpret_cast<uint32_t*>(&sm.vw[b][1][s][col]) = mid;
      *reinterpret_cast<uint32_t*>(&sm.vw[b][2][s][col]) = lo;
    }
  };

  auto output = [&](int c) {                   // the parts of the chunk's output come together
    const int b = c & 1, n = min(L, len - c * L);
    float* ob = p.o + (size_t)(row0 + c * L) * H * vdim + (size_t)h * vdim + colb;
#pragma unroll
    for (int r = aux >> 3; r < L; r += 16) {
      const int col = (aux & 7) * 4;
      float4 y = *reinterpret_cast<const float4*>(&sm.part[b][0][r][col]);
#pragma unroll
      for (int i = 1; i < WPR; ++i) {
        const float4 z = *reinterpret_cast<const float4*>(&sm.part[b][i][r][col]);
        y.x += z.x, y.y += z.y, y.z += z.z, y.w += z.w;
      }
      if (MLSTM) {
        float nq = sm.a[b][r] * sm.nq[b][r];
#pragma unroll
        for (int i = 0; i < WPR; ++i) nq += sm.rs[b][i][r];
        const float den = fmaxf(fabsf(nq * p.q_scale), sm.em[b][r]) + p.den_eps;
        y.x = y.x * p.q_scale / den, y.y = y.y * p.q_scale / den, y.z = y.z * p.q_scale / den, y.w = y.w * p.q_scale / den;
      }
      const int4 bad = *reinterpret_cast<const int4*>(&sm.bad[b][col]);
      if (r >= bad.x) y.x = NAN;
      if (r >= bad.y) y.y = NAN;
      if (r >= bad.z) y.z = NAN;
      if (r >= bad.w) y.w = NAN;
      if (r < n && colb + col < vdim) *reinterpret_cast<float4*>(ob + (size_t)r * H * vdim + col) = y;
    }
  };

  // ---- start: the state's columns into registers (transposed: row = column g of the slice, two neighbouring rows of S per register pair) and shared memory
  float S[2][NTU][4];
  const int d0 = warp * (DIM / MW);            // this warp's rows of the state
  float* Sb = p.St + (((size_t)slot * H + h) * vdim + colb) * DIM;
  auto publish = [&]() {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NTU; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t part[3];
          split3_finite(S[mt][nt][2 * e], S[mt][nt][2 * e + 1], part[0], part[1], part[2]);
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&sm.s[i][mt * 16 + g + 8 * e][d0 + nt * 8 + 2 * t4]) = part[i];
        }
  };
  if (warp < MW) {
#pragma unroll
    for (int i = 0; i < PIECES; ++i) fetch_qk(0, i);
    cp_async_commit();
  } else if (aux < 128) {
    fetch_v(0);
  }
  if (warp < MW) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NTU; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = mt * 16 + g + 8 * e;
          float2 v = make_float2(0.f, 0.f);
          if (colb + col < vdim) v = *reinterpret_cast<const float2*>(Sb + (size_t)col * DIM + d0 + nt * 8 + 2 * t4);
          S[mt][nt][2 * e] = v.x;
          S[mt][nt][2 * e + 1] = v.y;
        }
    publish();
    if (tid < 2 * COLS) sm.bad[tid / COLS][tid % COLS] = L;
  } else if (MLSTM && warp == MW + 4) {
    m = p.mst[(size_t)slot * H + h];
    read_gates(0);
    gates(0);
  } else {
    if (MLSTM) {
      for (int r = aux; r < DIM; r += 128) sm.n[r] = p.nst[((size_t)slot * H + h) * DIM + r];
    } else if (aux <= L) {
      double x = p.decay[h], y = 1.0;          // powers to fp32 rounding
      for (int e = aux; e; e >>= 1, x *= x)
        if (e & 1) y *= x;
      sm.pw[aux] = (float)y;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (warp >= MW && warp < MW + 4) weigh(0);
  __syncthreads();

  const int rb = warp < MW / 2 ? warp / WPR : RB - 1 - (warp - MW / 2) / WPR, share = warp % WPR;   // (contracting warps) row block, and which part of its work
  const int ks0 = warp < MW ? share_from<RB, WPR, KS>(rb, share) : 0, ks1 = warp < MW ? share_from<RB, WPR, KS>(rb, share + 1) : 0;
  const int la = lane & 7, i0 = (lane >> 3) & 1, i1 = lane >> 4;  // ldmatrix: row within a matrix, and the matrix's place in two directions
  for (int c = 0; c < chunks; ++c) {
    const int b = c & 1, n = min(L, len - c * L);
    const bool more = c + 1 < chunks;
    if (warp < MW) {
      const int blocks = (n + 15) >> 4;        // blocks of 16 tokens that hold any
      if (rb < blocks) {
        float acc[4][4] = {}, rest[4][4] = {}, sc[2][NB][2][4] = {};   // rest: what the lower parts give, small enough to stay in the tensor cores' sums
        // scores of this warp's blocks (rows rb, keys share, share + WPR, ..), and then its share of Q S
        if (share <= rb) {
#pragma unroll 4
          for (int ks = 0; ks < KS; ++ks) {
            uint32_t qf[4], kf[4];
            if (more && ks % (KS / PIECES) == 0) fetch_qk(c + 1, ks / (KS / PIECES));    // (then this chunk is a whole one: every warp comes by)
            ldsm_x4(smem_u32(&sm.q[b][rb * 16 + i0 * 8 + la][ks * 16 + i1 * 8]), qf);
#pragma unroll
            for (int j = 0; j < NB; ++j) {
              const int kblk = share + j * WPR;
              if (kblk > rb) continue;
              ldsm_x4(smem_u32(&sm.k[b][kblk * 16 + i1 * 8 + la][ks * 16 + i0 * 8]), kf);
              float st[2][4];
              mma_bf16_first(st[0], qf, kf[0], kf[1]);
              mma_bf16_first(st[1], qf, kf[2], kf[3]);
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float x = st[e >> 2][e & 3];
                if constexpr (few) {           // what the sum rounds off, exactly (Knuth's two-sum), in a sum of its own
                  float& sum = sc[0][j][e >> 2][e & 3];
                  const float next = sum + x, back = next - sum;
                  sc[1][j][e >> 2][e & 3] += (sum - (next - back)) + (x - back);
                  sum = next;
                } else {                                   // two chains: half the roundings each
                  sc[ks & 1][j][e >> 2][e & 3] += x;
                }
              }
            }
          }
        } else if (more) {                       // no scores for this warp
#pragma unroll 1
          for (int i = 0; i < PIECES; ++i) fetch_qk(c + 1, i);
        }
        cp_async_commit();
#pragma unroll 2
        for (int ks = ks0; ks < ks1; ++ks) {
          uint32_t qf[4];
          ldsm_x4(smem_u32(&sm.q[b][rb * 16 + i0 * 8 + la][ks * 16 + i1 * 8]), qf);
#pragma unroll
          for (int np = 0; np < 2; ++np) {
            float hi[2][4];
            uint32_t sf[3][4];
#pragma unroll
            for (int i = 0; i < 3; ++i) ldsm_x4(smem_u32(&sm.s[i][np * 16 + i1 * 8 + la][ks * 16 + i0 * 8]), sf[i]);
            mma_bf16_first(hi[0], qf, sf[0][0], sf[0][1]);
            mma_bf16_first(hi[1], qf, sf[0][2], sf[0][3]);
#pragma unroll
            for (int i = 2; i > 0; --i) {
              mma_bf16(rest[2 * np], qf, sf[i][0], sf[i][1]);
              mma_bf16(rest[2 * np + 1], qf, sf[i][2], sf[i][3]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[2 * np + (e >> 2)][e & 3] += hi[e >> 2][e & 3];
          }
        }
        const int ra = rb * 16 + g, rc = ra + 8;
        const float aa = MLSTM ? sm.a[b][ra] : sm.pw[ra + 1], ac = MLSTM ? sm.a[b][rc] : sm.pw[rc + 1];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          acc[nt][0] = (acc[nt][0] + rest[nt][0]) * aa;
          acc[nt][1] = (acc[nt][1] + rest[nt][1]) * aa;
          acc[nt][2] = (acc[nt][2] + rest[nt][2]) * ac;
          acc[nt][3] = (acc[nt][3] + rest[nt][3]) * ac;
#pragma unroll
          for (int e = 0; e < 4; ++e) rest[nt][e] = 0.f;
        }
        float suma = 0.f, sumc = 0.f;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          const int kblk = share + j * WPR;
          if (kblk > rb) continue;
          uint32_t pf[3][4];
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const int s = kblk * 16 + nt * 8 + 2 * t4;
            float* x = sc[0][j][nt];
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] += sc[1][j][nt][e];
            auto weight = [&](int t, int s_) { return MLSTM ? sm.D[b][t & 31][s_ & 31] : sm.pw[max(t - s_, 0)]; };
            x[0] = s <= ra ? x[0] * weight(ra, s) : 0.f;
            x[1] = s + 1 <= ra ? x[1] * weight(ra, s + 1) : 0.f;
            x[2] = s <= rc ? x[2] * weight(rc, s) : 0.f;
            x[3] = s + 1 <= rc ? x[3] * weight(rc, s + 1) : 0.f;
            suma += x[0] + x[1];
            sumc += x[2] + x[3];
            split3_finite(x[0], x[1], pf[0][2 * nt], pf[1][2 * nt], pf[2][2 * nt]);
            split3_finite(x[2], x[3], pf[0][2 * nt + 1], pf[1][2 * nt + 1], pf[2][2 * nt + 1]);
          }
#pragma unroll
          for (int np = 0; np < 2; ++np) {
            uint32_t vf[4];
            float hi[2][4];
            ldsm_x4_trans(smem_u32(&sm.v[b][kblk * 16 + i0 * 8 + la][np * 16 + i1 * 8]), vf);
            mma_bf16_first(hi[0], pf[0], vf[0], vf[1]);
            mma_bf16_first(hi[1], pf[0], vf[2], vf[3]);
#pragma unroll
            for (int i = 2; i > 0; --i) {
              mma_bf16(rest[2 * np], pf[i], vf[0], vf[1]);
              mma_bf16(rest[2 * np + 1], pf[i], vf[2], vf[3]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[2 * np + (e >> 2)][e & 3] += hi[e >> 2][e & 3];
          }
        }
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          *reinterpret_cast<float2*>(&sm.part[b][share][ra][nt * 8 + 2 * t4]) = make_float2(acc[nt][0] + rest[nt][0], acc[nt][1] + rest[nt][1]);
          *reinterpret_cast<float2*>(&sm.part[b][share][rc][nt * 8 + 2 * t4]) = make_float2(acc[nt][2] + rest[nt][2], acc[nt][3] + rest[nt][3]);
        }
        if (MLSTM) {
          suma += __shfl_xor_sync(0xffffffffu, suma, 1);
          suma += __shfl_xor_sync(0xffffffffu, suma, 2);
          sumc += __shfl_xor_sync(0xffffffffu, sumc, 1);
          sumc += __shfl_xor_sync(0xffffffffu, sumc, 2);
          if (t4 == 0) {
            sm.rs[b][share][ra] = suma;
            sm.rs[b][share][rc] = sumc;
          }
        }
      }
      // the update of this warp's rows of the state
      const float total = MLSTM ? sm.total[b] : sm.pw[n];
      float low[2][NTU][4] = {};
#pragma unroll
      for (int e = 0; e < 2 * NTU * 4; ++e) S[e / (NTU * 4)][e / 4 % NTU][e & 3] *= total;
#pragma unroll
      for (int kk = 0; kk < RB; ++kk) {
        if (kk >= blocks) break;
        uint32_t kf[NTU / 2][4];
#pragma unroll
        for (int np = 0; np < NTU / 2; ++np) ldsm_x4_trans(smem_u32(&sm.k[b][kk * 16 + i0 * 8 + la][d0 + np * 16 + i1 * 8]), kf[np]);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
          float hi[NTU][4];
          uint32_t vf[3][4];
#pragma unroll
          for (int i = 0; i < 3; ++i) ldsm_x4_trans(smem_u32(&sm.vw[b][i][kk * 16 + i1 * 8 + la][mt * 16 + i0 * 8]), vf[i]);
#pragma unroll
          for (int nt = 0; nt < NTU; ++nt) mma_bf16_first(hi[nt], vf[0], kf[nt / 2][(nt & 1) * 2], kf[nt / 2][(nt & 1) * 2 + 1]);
#pragma unroll
          for (int i = 2; i > 0; --i)
#pragma unroll
            for (int nt = 0; nt < NTU; ++nt) mma_bf16(low[mt][nt], vf[i], kf[nt / 2][(nt & 1) * 2], kf[nt / 2][(nt & 1) * 2 + 1]);
#pragma unroll
          for (int e = 0; e < NTU * 4; ++e) S[mt][e >> 2][e & 3] += hi[e >> 2][e & 3];
        }
      }
#pragma unroll
      for (int e = 0; e < 2 * NTU * 4; ++e) S[e / (NTU * 4)][e / 4 % NTU][e & 3] += low[e / (NTU * 4)][e / 4 % NTU][e & 3];
    } else if (MLSTM && warp == MW + 4) {
      if (more) gates(c + 1);
    } else {
      if (more) fetch_v(c + 1);
      if (c > 0) output(c - 1);
      if (MLSTM && more) asm volatile("bar.arrive 2, 160;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (aux < COLS) sm.bad[b ^ 1][aux] = L;
      if (MLSTM) {                             // q . n before the chunk, then n after it
        const int t = aux >> 2;
        float x = 0.f;
#pragma unroll 4
        for (int i = aux & 3; i < DIM / 8; i += 4) {
          float qv[8];
          unpack8(*reinterpret_cast<const uint4*>(&sm.q[b][t][i * 8]), qv);
#pragma unroll
          for (int e = 0; e < 8; ++e) x = fmaf(qv[e], sm.n[i * 8 + e], x);
        }
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        if ((aux & 3) == 0) sm.nq[b][t] = x;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (2 * aux < DIM) {
          float x0 = 0.f, x1 = 0.f;
#pragma unroll 4
          for (int s = 0; s < L; s += 4) {
            const float4 w = *reinterpret_cast<const float4*>(&sm.w[b][s]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float ws = i == 0 ? w.x : i == 1 ? w.y : i == 2 ? w.z : w.w;
              float k0, k1;
              unpack_bf16x2(*reinterpret_cast<const uint32_t*>(&sm.k[b][s + i][2 * aux]), k0, k1);
              x0 = fmaf(ws, k0, x0);
              x1 = fmaf(ws, k1, x1);
            }
          }
          sm.n[2 * aux] = fmaf(sm.total[b], sm.n[2 * aux], x0);
          sm.n[2 * aux + 1] = fmaf(sm.total[b], sm.n[2 * aux + 1], x1);
        }
      }
      if (more) {
        cp_async_wait<0>();                    // the helping warps' own copies: V
        if (MLSTM) asm volatile("bar.sync 3, 160;" ::: "memory");
        else asm volatile("bar.sync 1, 128;" ::: "memory");
        weigh(c + 1);
      }
    }
    cp_async_wait<0>();
    __syncthreads();                           // the chunk's contractions are done, the next chunk's inputs are there
    if (warp < MW) publish();
    __syncthreads();
  }
  if (warp >= MW && warp < MW + 4 && chunks > 0) output(chunks - 1);

  if (warp < MW) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < NTU; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = mt * 16 + g + 8 * e;
          if (colb + col < vdim) *reinterpret_cast<float2*>(Sb + (size_t)col * DIM + d0 + nt * 8 + 2 * t4) = make_float2(S[mt][nt][2 * e], S[mt][nt][2 * e + 1]);
        }
  } else if (MLSTM && blockIdx.x == 0) {       // the other CTAs of the head may not have read n and m yet
    float* n_out = p.ws ? p.ws + ((size_t)seg * H + h) * (DIM + 1) : p.nst + ((size_t)slot * H + h) * DIM;
    float* m_out = p.ws ? n_out + DIM : p.mst + (size_t)slot * H + h;
    if (warp < MW + 4)
      for (int r = aux; r < DIM; r += 128) n_out[r] = sm.n[r];
    else if (lane == 0) *m_out = m;
  }
}

template <bool MLSTM, int DIM, int L, bool few = false>
int launch_chunks(const ChunkArgs& p, int nseg, cudaStream_t stream) {
  const size_t smem = sizeof(ChunkSmem<DIM, L>);
  LIA_CUDA(cudaFuncSetAttribute(chunk_scan_kernel<MLSTM, DIM, L, few>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  lia_launch_after(chunk_scan_kernel<MLSTM, DIM, L, few>, dim3((p.vdim + COLS - 1) / COLS, p.H, nseg), dim3((MW + 4 + MLSTM) * 32), smem, stream, p);
  LIA_LAUNCH_CHECK();
  return LIA_OK;
}

bool whole_vectors(const ChunkArgs& p) {
  const uintptr_t in = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.o);
  return in % 16 == 0 && reinterpret_cast<uintptr_t>(p.St) % 8 == 0 && p.ldqk % 8 == 0 && p.ldv % 8 == 0 && p.vdim % 8 == 0;
}

}  // namespace

extern "C" int lia_chunk_scan_takes(int mlstm, int dim, int vdim) { return vdim > 0 && vdim % 8 == 0 && (dim == 128 || (mlstm && dim == 256)); }

extern "C" int lia_chunk_scan_rows() { return SHORT; }

extern "C" int lia_chunk_scan_few() { return FEW; }

extern "C" int lia_decay_scan_chunks(const void* q, const void* k, int ldqk, const void* v, int ldv, const float* decay, float* state_S, const int* segs, int nseg,
                                     int mixed, int H, int G, int dim, int vdim, float* o, lia_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LIA_CHECK_ARG(q && k && v && decay && state_S && segs && o, "lia_decay_scan_chunks: null pointer");
  LIA_CHECK_ARG(nseg > 0 && nseg <= 65535 && H > 0 && H <= 65535 && G > 0 && H % G == 0 && lia_chunk_scan_takes(0, dim, vdim),
                "lia_decay_scan_chunks: bad shape nseg=%d H=%d G=%d dim=%d vdim=%d", nseg, H, G, dim, vdim);
  ChunkArgs p{reinterpret_cast<const bf16*>(q), reinterpret_cast<const bf16*>(k), reinterpret_cast<const bf16*>(v), ldqk, ldv, decay, nullptr, state_S, nullptr,
              nullptr, nullptr, segs, H, G, vdim, 1.f, 0.f, o};
  LIA_CHECK_ARG(whole_vectors(p), "lia_decay_scan_chunks: rows are not whole 16-byte vectors");
  int rc = mixed & 4 ? LIA_OK : launch_chunks<false, 128, 64>(p, nseg, stream);
  if (rc == LIA_OK && !(mixed & 2)) rc = launch_chunks<false, 128, 64, true>(p, nseg, stream);
  return rc != LIA_OK || !(mixed & 1) ? rc : decay_scan_tokens(q, k, ldqk, v, ldv, decay, state_S, segs, SHORT, nseg, H, G, dim, vdim, o, stream);
}

extern "C" int lia_mlstm_scan_chunks(const void* q, const void* k, const void* v, int ld, const float* gates, float* state_S, float* state_n, float* state_m,
                                     const int* segs, int nseg, int mixed, int H, int dim, int vdim, float q_scale, float den_eps, float* o, float* ws,
                                     lia_stream_t stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  LIA_CHECK_ARG(q && k && v && gates && state_S && state_n && state_m && segs && o && ws, "lia_mlstm_scan_chunks: null pointer");
  LIA_CHECK_ARG(nseg > 0 && nseg <= 65535 && H > 0 && H <= 65535 && lia_chunk_scan_takes(1, dim, vdim), "lia_mlstm_scan_chunks: bad shape nseg=%d H=%d dim=%d vdim=%d",
                nseg, H, dim, vdim);
  ChunkArgs p{reinterpret_cast<const bf16*>(q), reinterpret_cast<const bf16*>(k), reinterpret_cast<const bf16*>(v), ld, ld, nullptr, gates, state_S, state_n, state_m,
              vdim > 16 ? ws : nullptr, segs, H, H, vdim, q_scale, den_eps, o};              // one column block (of either kernel): straight into the state
  LIA_CHECK_ARG(whole_vectors(p), "lia_mlstm_scan_chunks: rows are not whole 16-byte vectors");
  const int rc = dim == 128 ? launch_chunks<true, 128, 32>(p, nseg, stream) : launch_chunks<true, 256, 32>(p, nseg, stream);
  if (rc != LIA_OK) return rc;
  if (mixed) return mlstm_scan_tokens(q, k, v, ld, gates, state_S, state_n, state_m, ws, segs, SHORT, nseg, H, dim, vdim, q_scale, den_eps, o, stream);
  return p.ws ? mlstm_take_state(p.ws, segs, nseg, state_n, state_m, H, dim, stream) : LIA_OK;
}
