// Four neighbouring numbers of a row at a time, and a block's sum, for the row kernels.
#pragma once
#include "common.cuh"

namespace {

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  float4 f;
  unpack_bf16x2(u.x, f.x, f.y);
  unpack_bf16x2(u.y, f.z, f.w);
  return f;
}
__device__ __forceinline__ void store4(float* p, const float4& f) { *reinterpret_cast<float4*>(p) = f; }
__device__ __forceinline__ void store4(bf16* p, const float4& f) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(f.x, f.y), pack_bf16x2(f.z, f.w)); }
__device__ __forceinline__ float sum4(const float4& f) { return (f.x + f.y) + (f.z + f.w); }
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w); }

// Sum over 256 threads.  Each call of one kernel hands in a buffer of its own (8 floats), so one barrier is enough.
__device__ __forceinline__ float block_sum256(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  const float4 a = *reinterpret_cast<const float4*>(red), b = *reinterpret_cast<const float4*>(red + 4);
  return sum4(a) + sum4(b);
}

// whether rows of this stride, in numbers, start on whole vectors of 4 (host)
template <typename T> inline bool rows_of_4(const T* p, long long ld) { return reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0 && ld % 4 == 0; }

}  // namespace
