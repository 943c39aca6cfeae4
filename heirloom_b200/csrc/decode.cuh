// Pieces that the kernels of one-token steps share (decode.cu, decode_block.cu).
#pragma once
#include <cooperative_groups.h>

#include "kernels.h"

namespace hl {
namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ void cp_async16(void* shared, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(shared)), "l"(global) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T> __device__ __forceinline__ float as_f32(T x);
template <> __device__ __forceinline__ float as_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float as_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> struct Pack;  // sixteen bytes of weights
template <> struct Pack<float> {
  static constexpr int N = 4;
  __device__ static void unpack(const uint4& u, float (&v)[4]) {
    v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
  }
};
template <> struct Pack<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void unpack(const uint4& u, float (&v)[8]) {
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
};

constexpr int GV_SPAN = 1024;  // contraction elements a warp holds at a time, 32 a lane

template <int N> __device__ __forceinline__ void load_x(const float* p, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 t = *reinterpret_cast<const float4*>(p + i);
    v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
  }
}
template <int N> __device__ __forceinline__ void load_x(const __nv_bfloat16* p, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const uint2 t = *reinterpret_cast<const uint2*>(p + i);
    const float2 a = unpack_bf16x2(t.x), b = unpack_bf16x2(t.y);
    v[i] = a.x; v[i + 1] = a.y; v[i + 2] = b.x; v[i + 3] = b.y;
  }
}

}  // namespace
}  // namespace hl
