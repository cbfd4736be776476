// Four adjacent values of a storage plane at once.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dtsgb {

// Four consecutive storage values, kept packed until they are used.
template <typename TS>
struct Raw4;
template <>
struct Raw4<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) {
    v = __ldg(reinterpret_cast<const float4*>(p));
  }
  __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ float operator[](int k) const {
    return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
  }
};
template <>
struct Raw4<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    v = __ldg(reinterpret_cast<const uint2*>(p));
  }
  __device__ __forceinline__ void zero() { v = make_uint2(0u, 0u); }
  // bf16 -> f32 is exact: the 16 bits become the high half
  __device__ __forceinline__ float operator[](int k) const {
    const unsigned w = k < 2 ? v.x : v.y;
    return __uint_as_float((k & 1) ? (w & 0xffff0000u) : (w << 16));
  }
};

__device__ __forceinline__ float f4_get(const float4& v, int k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}
__device__ __forceinline__ unsigned u4_get(const uint4& v, int k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

}  // namespace dtsgb
