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

// The same 16 bytes (four fp32 or eight bf16 elements) at a time: `visit(fast, slow, x)`; a thread's elements have the same `fast`
// in every tile.
template <typename T>
constexpr int kChunk = 16 / static_cast<int>(sizeof(T));
template <typename T>
constexpr int kChunksPerRow = kTile / kChunk<T>;
template <typename T>
constexpr int kChunkRows = kThreads / kChunksPerRow<T>;      // rows of a tile that the CTA reads at once

__device__ __forceinline__ void unpack(const uint4& raw, float (&x)[4]) {
  x[0] = __uint_as_float(raw.x);
  x[1] = __uint_as_float(raw.y);
  x[2] = __uint_as_float(raw.z);
  x[3] = __uint_as_float(raw.w);
}
__device__ __forceinline__ void unpack(const uint4& raw, float (&x)[8]) {
  const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {      // a bf16 value is the upper half of the fp32 one
    x[2 * i] = __uint_as_float(words[i] << 16);
    x[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000u);
  }
}

template <typename T, typename Visit>
__device__ __forceinline__ void sweep_tile_chunks(const T* __restrict__ src, int64_t s_slow, int fast0, int slow0, int fast_end,
                                                  int slow_end, Visit visit) {
  constexpr int kRounds = kTile / kChunkRows<T>;
  const int offset = threadIdx.x % kChunksPerRow<T> * kChunk<T>, row = threadIdx.x / kChunksPerRow<T>;
  const int fast = fast0 + offset;
  uint4 raw[kRounds];
#pragma unroll
  for (int u = 0; u < kRounds; ++u) {
    const int slow = slow0 + row + u * kChunkRows<T>;
    raw[u] = make_uint4(0, 0, 0, 0);
    if (slow < slow_end && fast + kChunk<T> <= fast_end) raw[u] = *reinterpret_cast<const uint4*>(src + fast + slow * s_slow);
  }
#pragma unroll
  for (int u = 0; u < kRounds; ++u) {
    const int slow = slow0 + row + u * kChunkRows<T>;
    float x[kChunk<T>];
    unpack(raw[u], x);
    if (slow < slow_end && fast < fast_end && fast + kChunk<T> > fast_end) {
#pragma unroll
      for (int e = 0; e < kChunk<T>; ++e) x[e] = fast + e < fast_end ? load_one(src + fast + e + slow * s_slow) : 0.f;
    }
    visit(offset, row + u * kChunkRows<T>, x);
  }
}

// Whether a source can be read 16 bytes at a time along its fast axis.
template <typename T>
bool reads_chunks(const T* src, int64_t s_fast, int64_t s_slow, int n_slow) {
  return s_fast == 1 && (n_slow == 1 || s_slow % kChunk<T> == 0) && reinterpret_cast<uintptr_t>(src) % 16 == 0;
}

// Whether a source can be read two elements at a time along its fast axis.
template <typename T>
bool reads_pairs(const T* src, int64_t s_fast, int64_t s_slow, int n_slow) {
  return s_fast == 1 && (n_slow == 1 || s_slow % 2 == 0) && reinterpret_cast<uintptr_t>(src) % (2 * sizeof(T)) == 0;
}

}  // namespace sweep
}  // namespace soapb200
