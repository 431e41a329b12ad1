// 64 x 64 tiles of a strided matrix, read along its unit stride whichever way it lies (half_planes.cu, elementwise.cu).
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace soapb200 {
namespace sweep {

constexpr int kTile = 64;
constexpr int kThreads = 256;

__device__ __forceinline__ float load_one(const float* p) { return *p; }
__device__ __forceinline__ float load_one(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float2 load_two(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_two(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}

// The tile's elements, two along the source's fast axis per lane and step: `visit(fast, slow, x0, x1)` with offsets inside
// the tile; elements outside the matrix are zero.
template <typename T, typename Visit>
__device__ __forceinline__ void sweep_tile(const T* __restrict__ src, int64_t s_fast, int64_t s_slow, int fast0, int slow0,
                                           int fast_end, int slow_end, bool pairs, Visit visit) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fast = fast0 + 2 * lane;
  float2 x[kTile / 8];
#pragma unroll
  for (int u = 0; u < kTile / 8; ++u) {
    const int slow = slow0 + warp + 8 * u;
    x[u] = make_float2(0.f, 0.f);
    if (slow < slow_end && fast < fast_end) {
      const T* at = src + fast * s_fast + slow * s_slow;
      if (pairs && fast + 1 < fast_end) {
        x[u] = load_two(at);
      } else {
        x[u].x = load_one(at);
        if (fast + 1 < fast_end) x[u].y = load_one(at + s_fast);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kTile / 8; ++u) visit(2 * lane, warp + 8 * u, x[u].x, x[u].y);
}

// Whether a source can be read two elements at a time along its fast axis.
template <typename T>
bool reads_pairs(const T* src, int64_t s_fast, int64_t s_slow, int n_slow) {
  return s_fast == 1 && (n_slow == 1 || s_slow % 2 == 0) && reinterpret_cast<uintptr_t>(src) % (2 * sizeof(T)) == 0;
}

}  // namespace sweep
}  // namespace soapb200
