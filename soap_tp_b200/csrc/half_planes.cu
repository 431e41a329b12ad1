// Scaled fp16 operand planes (gemm_half.h) of a matrix, in one or both orientations.
//
// Bound by memory: the source is read twice (once for the largest magnitude of every row and column, once to convert it)
// and each wanted plane written once.  64 x 64 tiles, turned in shared memory, so that reads run along the source's unit
// stride and writes along each plane's, whichever way the source lies.
//
// With a RangeGuard the second pass also decides whether fp16 pairs hold the matrix and, where they do not, writes the mixed
// form of the matrix and of its bases.  That takes no launch of its own: there is about one CTA per SM more, which looks at the
// largest magnitude of every row and column (64 KB from L2 at 8192 x 8192) while the others convert.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <stdexcept>
#include <string>
#include <type_traits>

#include "gemm_half.h"
#include "launch_util.h"
#include "split_write.cuh"
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

// What the second pass writes beside the planes where fp16 pairs do not hold the matrix: the mixed form of it and its bases.
struct MixedJob {
  const void* src;
  int64_t s_fast, s_slow;
  int n_fast, n_slow;              // 0: nothing to do
  bool pairs, along_pairs, across_pairs;
  SplitTarget along, across;
};
struct MixedWork {
  int* wide;
  const uint32_t* maxima[2];
  int counts[2];
  int nearest;
  int rows;                        // rows of CTAs that do it
  MixedJob matrix, bases[2];
};
struct NoWork {};
template <bool DECIDED>
using Work = std::conditional_t<DECIDED, MixedWork, NoWork>;

template <typename T>
__device__ __forceinline__ void write_mixed(const MixedJob& job, float (*tile)[kTile + 1], int helper, int helpers, int nearest) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles_fast = (job.n_fast + kTile - 1) / kTile, tiles = tiles_fast * ((job.n_slow + kTile - 1) / kTile);
  for (int t = helper; t < tiles; t += helpers) {
    const int fast0 = t % tiles_fast * kTile, slow0 = t / tiles_fast * kTile;
    __syncthreads();                                 // the tile before has been written out
    sweep_tile(static_cast<const T*>(job.src), job.s_fast, job.s_slow, fast0, slow0, job.n_fast, job.n_slow, job.pairs,
               [&](int fast, int slow, float x0, float x1) {
                 tile[slow][fast] = x0;
                 tile[slow][fast + 1] = x1;
               });
    __syncthreads();
    if (job.along.hi && fast0 + 2 * lane < job.n_fast)
      for (int s = warp; s < kTile && slow0 + s < job.n_slow; s += 8)
        write_split(job.along, job.along_pairs, fast0 + 2 * lane, slow0 + s, job.n_fast, tile[s][2 * lane],
                    tile[s][2 * lane + 1], nearest);
    if (job.across.hi && slow0 + 2 * lane < job.n_slow)
      for (int f = warp; f < kTile && fast0 + f < job.n_fast; f += 8)
        write_split(job.across, job.across_pairs, slow0 + 2 * lane, fast0 + f, job.n_slow, tile[2 * lane][f],
                    tile[2 * lane + 1][f], nearest);
  }
}

// RangeGuard's decision, the same in every CTA that asks.
__device__ __forceinline__ bool too_wide(const MixedWork& work, uint32_t* scratch) {
  uint32_t most = 0, least = 0xffffffffu;
  for (int a = 0; a < 2; ++a) {
    for (int i = threadIdx.x; i < work.counts[a]; i += kThreads) {
      const uint32_t word = work.maxima[a][i];
      most = max(most, word);
      least = min(least, word);
    }
  }
  most = __reduce_max_sync(0xffffffffu, most);
  least = __reduce_min_sync(0xffffffffu, least);
  if ((threadIdx.x & 31) == 0) {
    scratch[threadIdx.x >> 5] = most;
    scratch[kThreads / 32 + (threadIdx.x >> 5)] = least;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    most = max(most, scratch[w]);
    least = min(least, scratch[kThreads / 32 + w]);
  }
  const int top = static_cast<int>(most >> 23), bottom = static_cast<int>(least >> 23);
  return most != 0 && (least == 0 || top == 255 || top - bottom > kRangeOrders);       // (a matrix of zeros is held)
}

// Out of line: the rarely taken path must not cost the other one registers.
template <typename T>
__device__ __noinline__ void help(const MixedWork& work, float (*tile)[kTile + 1], int helper, int helpers) {
  const bool wide = too_wide(work, reinterpret_cast<uint32_t*>(tile));
  if (helper == 0 && threadIdx.x == 0) *work.wide = wide;
  if (!wide) return;
  write_mixed<T>(work.matrix, tile, helper, helpers, work.nearest);
  write_mixed<float>(work.bases[0], tile, helper, helpers, work.nearest);
  write_mixed<float>(work.bases[1], tile, helper, helpers, work.nearest);
}

// `along`: depth runs along the source's fast axis; `across`: depth runs along its slow axis.  The first rows of CTAs are there
// for the decision and the mixed form (DECIDED); eight CTAs per SM, so that their registers do not cost the others occupancy (with the 48 that
// they ask for the planes of 4096^2 fp32 took 65 us instead of 59).
template <typename T, bool DECIDED>
__global__ void __launch_bounds__(kThreads, DECIDED ? 8 : 1) half_planes_kernel(const T* __restrict__ src, int64_t s_fast, int64_t s_slow,
                                                               int n_fast, int n_slow, bool pairs, const HalfTarget along,
                                                               const HalfTarget across, const __grid_constant__ Work<DECIDED> work) {
  __shared__ float tile[kTile][kTile + 1];           // [slow][fast]
  __shared__ float up_along[kTile], up_across[kTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  wait_for_predecessor();
  let_successor_start();
  int tile_row = blockIdx.y;
  if constexpr (DECIDED) {
    tile_row -= work.rows;
    if (tile_row < 0) {
      help<T>(work, tile, blockIdx.y * gridDim.x + blockIdx.x, work.rows * gridDim.x);
      return;
    }
  }
  const int fast0 = blockIdx.x * kTile, slow0 = tile_row * kTile;
  if (threadIdx.x < kTile) {
    const int slow = slow0 + threadIdx.x;
    if (along.h && slow < n_slow) {
      const HalfScale s = half_scale(along.largest[slow]);
      up_along[threadIdx.x] = s.multiplier;
      if (fast0 == 0) along.scale[slow] = s.inverse;
    }
  } else if (threadIdx.x < 2 * kTile) {
    const int f = threadIdx.x - kTile, fast = fast0 + f;
    if (across.h && fast < n_fast) {
      const HalfScale s = half_scale(across.largest[fast]);
      up_across[f] = s.multiplier;
      if (slow0 == 0) across.scale[fast] = s.inverse;
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

bool fast_is_first(int64_t s_i, int64_t s_j, int rows, int cols) {
  return cols == 1 || (rows > 1 && s_i <= s_j);      // the axis with the smaller stride is swept by the lanes
}

template <typename T>
MixedJob mixed_job(const T* src, int64_t s_fast, int64_t s_slow, int n_fast, int n_slow, const SplitTarget& along,
                   const SplitTarget& across) {
  return MixedJob{src, s_fast, s_slow, n_fast, n_slow, reads_pairs(src, s_fast, s_slow, n_slow), writes_pairs(along),
                  writes_pairs(across), along, across};
}

MixedJob basis_job(const WideBasis& b) {
  if (!b.src) return MixedJob{};
  return fast_is_first(b.s_i, b.s_j, b.size, b.size) ? mixed_job(b.src, b.s_i, b.s_j, b.size, b.size, b.plain, b.turned)
                                                     : mixed_job(b.src, b.s_j, b.s_i, b.size, b.size, b.turned, b.plain);
}

template <typename T>
void launch(const T* src, int64_t s_fast, int64_t s_slow, int n_fast, int n_slow, const HalfTarget& along,
            const HalfTarget& across, const SplitTarget& mixed_along, const SplitTarget& mixed_across, const RangeGuard& guard,
            cudaStream_t stream) {
  const bool pairs = reads_pairs(src, s_fast, s_slow, n_slow);
  if (along.largest) check(cudaMemsetAsync(along.largest, 0, sizeof(uint32_t) * n_slow, stream), "half_planes");
  if (across.largest) check(cudaMemsetAsync(across.largest, 0, sizeof(uint32_t) * n_fast, stream), "half_planes");
  const int tiles_fast = (n_fast + kTile - 1) / kTile, tiles_slow = (n_slow + kTile - 1) / kTile;
  // enough CTAs for every SM several times over before a CTA takes more than one tile
  int strip = static_cast<int>(static_cast<int64_t>(tiles_fast) * tiles_slow / (148 * 8));
  strip = strip < 1 ? 1 : (strip > 16 ? 16 : strip);
  const int helper_rows = guard.wide ? (148 + tiles_fast - 1) / tiles_fast : 0;
  const dim3 strips(tiles_fast, (tiles_slow + strip - 1) / strip), tiles(tiles_fast, tiles_slow + helper_rows);
  if (strips.y > 65535 || tiles.y > 65535) throw std::invalid_argument("half_planes: matrix too long");
  check(launch_dependent(largest_kernel<T>, strips, dim3(kThreads), 0, stream, src, s_fast, s_slow, n_fast, n_slow, strip, pairs,
                         across.largest, along.largest),
        "largest_kernel");
  auto convert = [&](auto kernel, const auto& work) {
    check(launch_dependent(kernel, tiles, dim3(kThreads), 0, stream, src, s_fast, s_slow, n_fast, n_slow, pairs, along, across, work),
          "half_planes_kernel");
  };
  if (guard.wide)
    convert(half_planes_kernel<T, true>,
            MixedWork{guard.wide, {along.largest, across.largest}, {n_slow, n_fast}, guard.nearest, helper_rows, mixed_job(src, s_fast, s_slow, n_fast, n_slow, mixed_along, mixed_across),
                      {basis_job(guard.bases[0]), basis_job(guard.bases[1])}});
  else
    convert(half_planes_kernel<T, false>, NoWork{});
}

}  // namespace

void half_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const HalfTarget& plain,
                 const HalfTarget& turned, const RangeGuard& guard, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || (!plain.h && !turned.h)) return;
  for (const HalfTarget* t : {&plain, &turned}) {
    if (t->h && (!t->largest || t->ld % 64 != 0 || t->ld < (t == &plain ? rows : cols) ||
                 (reinterpret_cast<uintptr_t>(t->h) & 15) != 0 || (reinterpret_cast<uintptr_t>(t->l) & 15) != 0))
      throw std::invalid_argument("half_planes: planes need 16-byte alignment and a pitch that is a multiple of 64");
    if (guard.wide && !t->largest)
      throw std::invalid_argument("half_planes: a decision on the range needs the maxima of both orientations");
  }
  const bool rows_fast = fast_is_first(s_i, s_j, rows, cols);
  auto go = [&](auto* typed) {
    if (rows_fast) launch(typed, s_i, s_j, rows, cols, plain, turned, guard.mixed, SplitTarget{}, guard, stream);
    else launch(typed, s_j, s_i, cols, rows, turned, plain, SplitTarget{}, guard.mixed, guard, stream);
  };
  if (source_type == 0) go(static_cast<const float*>(src));
  else if (source_type == 1) go(static_cast<const __nv_bfloat16*>(src));
  else throw std::invalid_argument("half_planes: unknown source type");
}

}  // namespace soapb200
