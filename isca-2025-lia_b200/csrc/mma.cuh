// Warp-level tensor-core helpers (mma.sync m16n8k16 bf16 with fp32 sums, ldmatrix, cp.async) shared by the kernels whose operands
// are made in registers between two contractions, and the exact split of an fp32 number into three bf16 numbers.
//
// Splitting: x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi), lo = bf16(x - hi - mid).  Both differences are exact, and 3 x 8
// significant bits hold the 24 of an fp32 number, so an fp32 operand times a bf16 operand is three bf16 products with fp32
// sums: the precision of the fp32 FMA chain it replaces.
#pragma once
#include "common.cuh"

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// c += a (16 x 16) b (16 x 8).  Lane l = 4 g + t holds a: rows g, g + 8 at columns 2t, 2t + 1 (a[0], a[1]) and 2t + 8, 2t + 9 (a[2], a[3]);
// b: rows 2t, 2t + 1 (b0) and 2t + 8, 2t + 9 (b1) of column g; c: row g, columns 2t, 2t + 1 (c[0], c[1]) and row g + 8 (c[2], c[3]).
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c = a b
__device__ __forceinline__ void mma_bf16_first(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// 16 bytes global -> shared; `n` < 16 bytes are read and the rest is zero
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// two neighbouring fp32 numbers as three packed bf16 pairs; an infinity stays one (its remainders would be NaN)
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  float hx, hy;
  unpack_bf16x2(hi, hx, hy);
  const float rx = fabsf(hx) == INFINITY ? 0.f : x - hx, ry = fabsf(hy) == INFINITY ? 0.f : y - hy;
  mid = pack_bf16x2(rx, ry);
  float mx, my;
  unpack_bf16x2(mid, mx, my);
  lo = pack_bf16x2(rx - mx, ry - my);
}
// the same for finite numbers
__device__ __forceinline__ void split3_finite(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(x, y);
  float hx, hy, mx, my;
  unpack_bf16x2(hi, hx, hy);
  const float rx = x - hx, ry = y - hy;
  mid = pack_bf16x2(rx, ry);
  unpack_bf16x2(mid, mx, my);
  lo = pack_bf16x2(rx - mx, ry - my);
}
