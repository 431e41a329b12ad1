// Writing elements of an operand as tf32 value and remainder (elementwise.cu, half_planes.cu).
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "elementwise.h"
#include "gemm.h"

namespace soapb200 {

__device__ __forceinline__ float tf32_hi(float x, int nearest) {
  if (nearest) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
  }
  return __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
}

__device__ __forceinline__ uint16_t bf16_bits(float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  return *reinterpret_cast<const uint16_t*>(&b);
}

// Elements i, i + 1 of column j of an operand of depth n; nothing past the depth is written (the planes may be a window).
__device__ __forceinline__ void write_split(const SplitTarget& to, bool pairs, int64_t i, int64_t j, int n, float x0, float x1,
                                            int nearest) {
  const float h0 = tf32_hi(x0, nearest), h1 = tf32_hi(x1, nearest);
  const int64_t at = i + j * to.ldo, at16 = to.hl ? bf16_plane_index(i) + j * to.ld16 : 0;
  if (pairs && i + 1 < n) {
    *reinterpret_cast<float2*>(to.hi + at) = make_float2(h0, h1);
    if (to.hl) {
      *reinterpret_cast<__nv_bfloat162*>(to.hl + at16) = __floats2bfloat162_rn(x0, x1);
      *reinterpret_cast<__nv_bfloat162*>(to.hl + at16 + 32) = __floats2bfloat162_rn(x0 - h0, x1 - h1);
    } else {
      *reinterpret_cast<float2*>(to.lo + at) = make_float2(x0 - h0, x1 - h1);
    }
    return;
  }
  for (int e = 0; e < 2 && i + e < n; ++e) {
    const float x = e ? x1 : x0, h = e ? h1 : h0;
    to.hi[at + e] = h;
    if (to.hl) {         // i is even, so that i and i + 1 are neighbours in the interleaved plane too
      to.hl[at16 + e] = bf16_bits(x);
      to.hl[at16 + e + 32] = bf16_bits(x - h);
    } else {
      to.lo[at + e] = x - h;
    }
  }
}

// Whether a target takes two elements at a time along its depth.
inline bool writes_pairs(const SplitTarget& t) {
  return (reinterpret_cast<uintptr_t>(t.hi) & 7) == 0 && t.ldo % 2 == 0 &&
         (t.hl ? (reinterpret_cast<uintptr_t>(t.hl) & 3) == 0 && t.ld16 % 2 == 0 : (reinterpret_cast<uintptr_t>(t.lo) & 7) == 0);
}

}  // namespace soapb200
