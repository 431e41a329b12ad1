// Scaled fp16 operand planes (gemm_half.h) of a matrix, in one or both orientations.
//
// Bound by memory: the source is read twice (once for the largest magnitude of every row and column, once to convert it)
// and each wanted plane written once.  64 x 64 tiles, turned in shared memory, so that reads run along the source's unit
// stride and writes along each plane's, whichever way the source lies.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <stdexcept>
#include <string>

#include "gemm_half.h"
#include "launch_util.h"
#include "tile_sweep.cuh"

namespace soapb200 {
namespace {

using namespace sweep;

__device__ __forceinline__ uint32_t magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// Largest magnitude (as a bit pattern, which orders like the value) along the fast and the slow axis.  A CTA walks
// `strip` tiles along the slow axis and keeps the maxima of its fast-axis elements in registers meanwhile.
template <typename T>
__global__ void __launch_bounds__(kThreads) largest_kernel(const T* __restrict__ src, int64_t s_fast, int64_t s_slow, int n_fast,
                                                           int n_slow, int strip, bool pairs, uint32_t* __restrict__ of_fast,
                                                           uint32_t* __restrict__ of_slow) {
  __shared__ uint32_t fast_max[8][kTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fast0 = blockIdx.x * kTile;
  wait_for_predecessor();
  let_successor_start();
  uint32_t mine0 = 0, mine1 = 0;
  for (int t = 0; t < strip; ++t) {
    const int slow0 = (blockIdx.y * strip + t) * kTile;
    if (slow0 >= n_slow) break;
    sweep_tile(src, s_fast, s_slow, fast0, slow0, n_fast, n_slow, pairs, [&](int, int slow, float x0, float x1) {
      const uint32_t a = magnitude(x0), b = magnitude(x1);
      mine0 = max(mine0, a);
      mine1 = max(mine1, b);
      if (of_slow) {
        const uint32_t row = __reduce_max_sync(0xffffffffu, max(a, b));
        if (lane == 0 && slow0 + slow < n_slow) atomicMax(of_slow + slow0 + slow, row);
      }
    });
  }
  if (!of_fast) return;
  fast_max[warp][2 * lane] = mine0;
  fast_max[warp][2 * lane + 1] = mine1;
  __syncthreads();
  if (threadIdx.x < kTile && fast0 + threadIdx.x < n_fast) {
    uint32_t most = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) most = max(most, fast_max[w][threadIdx.x]);
    atomicMax(of_fast + fast0 + threadIdx.x, most);
  }
}

__device__ __forceinline__ void write_pair(const HalfTarget& to, int64_t at, float x0, float x1) {
  const __half2 h = __floats2half2_rn(x0, x1);
  *reinterpret_cast<__half2*>(to.h + at) = h;
  if (to.l) {
    const float2 back = __half22float2(h);
    *reinterpret_cast<__half2*>(to.l + at) = __floats2half2_rn(x0 - back.x, x1 - back.y);
  }
}

// `along`: depth runs along the source's fast axis; `across`: depth runs along its slow axis.
template <typename T>
__global__ void __launch_bounds__(kThreads) half_planes_kernel(const T* __restrict__ src, int64_t s_fast, int64_t s_slow,
                                                               int n_fast, int n_slow, bool pairs, const HalfTarget along,
                                                               const HalfTarget across) {
  __shared__ float tile[kTile][kTile + 1];           // [slow][fast]
  __shared__ float up_along[kTile], up_across[kTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fast0 = blockIdx.x * kTile, slow0 = blockIdx.y * kTile;
  wait_for_predecessor();
  let_successor_start();
  if (threadIdx.x < kTile) {
    const int slow = slow0 + threadIdx.x;
    if (along.h && slow < n_slow) {
      const HalfScale s = half_scale(along.largest[slow]);
      up_along[threadIdx.x] = s.multiplier;
      if (blockIdx.x == 0) along.scale[slow] = s.inverse;
    }
  } else if (threadIdx.x < 2 * kTile) {
    const int f = threadIdx.x - kTile, fast = fast0 + f;
    if (across.h && fast < n_fast) {
      const HalfScale s = half_scale(across.largest[fast]);
      up_across[f] = s.multiplier;
      if (blockIdx.y == 0) across.scale[fast] = s.inverse;
    }
  }
  sweep_tile(src, s_fast, s_slow, fast0, slow0, n_fast, n_slow, pairs, [&](int fast, int slow, float x0, float x1) {
    tile[slow][fast] = x0;
    tile[slow][fast + 1] = x1;
  });
  __syncthreads();
  // pitches are multiples of 64, so the second half of a pair that ends the depth lands in the padding
  if (along.h && fast0 + 2 * lane < n_fast) {
    for (int s = warp; s < kTile && slow0 + s < n_slow; s += 8)
      write_pair(along, fast0 + 2 * lane + (slow0 + s) * along.ld, tile[s][2 * lane] * up_along[s],
                 tile[s][2 * lane + 1] * up_along[s]);
  }
  if (across.h && slow0 + 2 * lane < n_slow) {
    for (int f = warp; f < kTile && fast0 + f < n_fast; f += 8)
      write_pair(across, slow0 + 2 * lane + (fast0 + f) * across.ld, tile[2 * lane][f] * up_across[f],
                 tile[2 * lane + 1][f] * up_across[f]);
  }
}

void check(cudaError_t err, const char* what) {
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(err));
}

template <typename T>
void launch(const T* src, int64_t s_fast, int64_t s_slow, int n_fast, int n_slow, const HalfTarget& along,
            const HalfTarget& across, cudaStream_t stream) {
  const bool pairs = reads_pairs(src, s_fast, s_slow, n_slow);
  if (along.h) check(cudaMemsetAsync(along.largest, 0, sizeof(uint32_t) * n_slow, stream), "half_planes");
  if (across.h) check(cudaMemsetAsync(across.largest, 0, sizeof(uint32_t) * n_fast, stream), "half_planes");
  const int tiles_fast = (n_fast + kTile - 1) / kTile, tiles_slow = (n_slow + kTile - 1) / kTile;
  // enough CTAs for every SM several times over before a CTA takes more than one tile
  int strip = static_cast<int>(static_cast<int64_t>(tiles_fast) * tiles_slow / (148 * 8));
  strip = strip < 1 ? 1 : (strip > 16 ? 16 : strip);
  const dim3 strips(tiles_fast, (tiles_slow + strip - 1) / strip), tiles(tiles_fast, tiles_slow);
  if (strips.y > 65535 || tiles.y > 65535) throw std::invalid_argument("half_planes: matrix too long");
  check(launch_dependent(largest_kernel<T>, strips, dim3(kThreads), 0, stream, src, s_fast, s_slow, n_fast, n_slow, strip, pairs,
                         across.h ? across.largest : nullptr, along.h ? along.largest : nullptr),
        "largest_kernel");
  check(launch_dependent(half_planes_kernel<T>, tiles, dim3(kThreads), 0, stream, src, s_fast, s_slow, n_fast, n_slow, pairs,
                         along, across),
        "half_planes_kernel");
}

}  // namespace

void half_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const HalfTarget& plain,
                 const HalfTarget& turned, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || (!plain.h && !turned.h)) return;
  for (const HalfTarget* t : {&plain, &turned})
    if (t->h && (t->ld % 64 != 0 || t->ld < (t == &plain ? rows : cols) || (reinterpret_cast<uintptr_t>(t->h) & 15) != 0 ||
                 (reinterpret_cast<uintptr_t>(t->l) & 15) != 0))
      throw std::invalid_argument("half_planes: planes need 16-byte alignment and a pitch that is a multiple of 64");
  const bool rows_fast = cols == 1 || (rows > 1 && s_i <= s_j);       // the axis with the smaller stride is swept by the lanes
  auto go = [&](auto* typed) {
    if (rows_fast) launch(typed, s_i, s_j, rows, cols, plain, turned, stream);
    else launch(typed, s_j, s_i, cols, rows, turned, plain, stream);
  };
  if (source_type == 0) go(static_cast<const float*>(src));
  else if (source_type == 1) go(static_cast<const __nv_bfloat16*>(src));
  else throw std::invalid_argument("half_planes: unknown source type");
}

}  // namespace soapb200
