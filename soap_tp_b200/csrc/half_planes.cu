// Scaled fp16 operand planes (gemm_half.h) of a matrix, in one or both orientations.
//
// Bound by memory: the source is read twice (once for the largest magnitude of every row and column, once to convert it)
// and each wanted plane written once.  64 x 64 tiles, turned in shared memory, so that reads run along the source's unit
// stride and writes along each plane's, whichever way the source lies; 16 bytes a thread, the reads where the source is aligned to
// that (the planes always are).  Two elements a thread kept too few bytes in flight for 16-bit sources
// (32064 x 2048 bf16, one orientation, 131 MB read twice and written once: 231 us, now 100; both orientations 128 us.  8192 x 8192 fp32, both:
// 205 us, 1.07 GB.)
//
// With a RangeGuard the second pass also decides whether fp16 pairs hold the matrix and, where they do not, writes the mixed
// form of the matrix and of its bases.  That takes no launch of its own: there is about one CTA per SM more, which looks at the
// largest magnitude of every row and column (64 KB from L2 at 8192 x 8192) while the others convert.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
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

// Scratch of the largest magnitudes back to zero.  A kernel, so that the chain of dependent launches goes through it; a memset
// of each array would stand between two of them.
template <int N>
struct ClearGroup {
  uint32_t* words[2 * N];
  int counts[2 * N];
};
template <int N>
__global__ void __launch_bounds__(kThreads) clear_kernel(const __grid_constant__ ClearGroup<N> group) {
  wait_for_predecessor();
  let_successor_start();
  uint32_t* words = group.words[blockIdx.y];
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < group.counts[blockIdx.y]; i += gridDim.x * kThreads) words[i] = 0;
}

// A matrix as the two passes over it see it.
struct Source {
  const void* src;
  int64_t s_fast, s_slow;
  int n_fast, n_slow, tiles_fast;
  bool pairs, chunks;      // may be read two elements, 16 bytes at a time
};
struct LargestJob {
  Source from;
  int strip;
  uint32_t *of_fast, *of_slow;
};
template <int N>
struct LargestGroup {
  LargestJob jobs[N];
  GroupBlocks<N> blocks;
};

// Largest magnitude (as a bit pattern, which orders like the value) along the fast and the slow axis.  A CTA walks
// `strip` tiles along the slow axis and keeps the maxima of its fast-axis elements in registers meanwhile.
template <typename T, int N>
__global__ void __launch_bounds__(kThreads) largest_kernel(const __grid_constant__ LargestGroup<N> group) {
  __shared__ uint32_t fast_max[kChunkRows<T>][kTile];      // (of the 8 warps where the source is read by pairs)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int member = group.blocks.member(blockIdx.x), block = blockIdx.x - group.blocks.first(member);
  const LargestJob& job = group.jobs[member];
  const T* src = static_cast<const T*>(job.from.src);
  const int n_fast = job.from.n_fast, n_slow = job.from.n_slow, strip = job.strip;
  uint32_t *of_fast = job.of_fast, *of_slow = job.of_slow;
  const int fast0 = block % job.from.tiles_fast * kTile, strip0 = block / job.from.tiles_fast * strip;
  wait_for_predecessor();
  let_successor_start();
  if (job.from.chunks) {
    constexpr int kAcross = kChunksPerRow<T>;      // threads that share a row
    const int row = threadIdx.x / kAcross, offset = threadIdx.x % kAcross * kChunk<T>;
    uint32_t mine[kChunk<T>] = {};
    for (int t = 0; t < strip; ++t) {
      const int slow0 = (strip0 + t) * kTile;
      if (slow0 >= n_slow) break;
      sweep_tile_chunks(src, job.from.s_slow, fast0, slow0, n_fast, n_slow, [&](int, int slow, const float (&x)[kChunk<T>]) {
        uint32_t most = 0;
#pragma unroll
        for (int e = 0; e < kChunk<T>; ++e) {
          const uint32_t a = magnitude(x[e]);
          mine[e] = max(mine[e], a);
          most = max(most, a);
        }
        if (of_slow) {
#pragma unroll
          for (int lanes = 1; lanes < kAcross; lanes *= 2) most = max(most, __shfl_xor_sync(0xffffffffu, most, lanes));
          if (threadIdx.x % kAcross == 0 && slow0 + slow < n_slow) atomicMax(of_slow + slow0 + slow, most);
        }
      });
    }
    if (!of_fast) return;
#pragma unroll
    for (int e = 0; e < kChunk<T>; ++e) fast_max[row][offset + e] = mine[e];
    __syncthreads();
    if (threadIdx.x < kTile && fast0 + threadIdx.x < n_fast) {
      uint32_t most = 0;
#pragma unroll
      for (int r = 0; r < kChunkRows<T>; ++r) most = max(most, fast_max[r][threadIdx.x]);
      atomicMax(of_fast + fast0 + threadIdx.x, most);
    }
    return;
  }
  uint32_t mine0 = 0, mine1 = 0;
  for (int t = 0; t < strip; ++t) {
    const int slow0 = (strip0 + t) * kTile;
    if (slow0 >= n_slow) break;
    sweep_tile(src, job.from.s_fast, job.from.s_slow, fast0, slow0, n_fast, n_slow, job.from.pairs, [&](int, int slow, float x0, float x1) {
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

// Eight elements along the depth of a plane, 16-byte aligned: `x(e)` the e-th.
template <typename Element>
__device__ __forceinline__ void write_eight(const HalfTarget& to, int64_t at, Element x) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x0 = x(2 * i), x1 = x(2 * i + 1);
    const __half2 high = __floats2half2_rn(x0, x1);
    const float2 back = __half22float2(high);
    const __half2 low = __floats2half2_rn(x0 - back.x, x1 - back.y);
    h[i] = *reinterpret_cast<const uint32_t*>(&high);
    l[i] = *reinterpret_cast<const uint32_t*>(&low);
  }
  *reinterpret_cast<uint4*>(to.h + at) = make_uint4(h[0], h[1], h[2], h[3]);
  if (to.l) *reinterpret_cast<uint4*>(to.l + at) = make_uint4(l[0], l[1], l[2], l[3]);
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
template <bool DECIDED>
struct PlaneJob {
  Source from;
  HalfTarget along, across;
  Work<DECIDED> work;
};
template <bool DECIDED, int N>
struct PlaneGroup {
  PlaneJob<DECIDED> jobs[N];
  GroupBlocks<N> blocks;
};
template <typename T, bool DECIDED, int N>
__global__ void __launch_bounds__(kThreads, DECIDED ? 8 : 1) half_planes_kernel(const __grid_constant__ PlaneGroup<DECIDED, N> group) {
  __shared__ float tile[kTile][kTile + 1];           // [slow][fast]
  __shared__ float up_along[kTile], up_across[kTile];
  const int member = group.blocks.member(blockIdx.x), block = blockIdx.x - group.blocks.first(member);
  const PlaneJob<DECIDED>& job = group.jobs[member];
  const int n_fast = job.from.n_fast, n_slow = job.from.n_slow;
  const HalfTarget along = job.along, across = job.across;
  wait_for_predecessor();
  let_successor_start();
  int tile_row = block / job.from.tiles_fast;
  if constexpr (DECIDED) {
    tile_row -= job.work.rows;
    if (tile_row < 0) {
      help<T>(job.work, tile, block, job.work.rows * job.from.tiles_fast);
      return;
    }
  }
  const int fast0 = block % job.from.tiles_fast * kTile, slow0 = tile_row * kTile;
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
  const T* src = static_cast<const T*>(job.from.src);
  if (job.from.chunks) {
    sweep_tile_chunks(src, job.from.s_slow, fast0, slow0, n_fast, n_slow, [&](int fast, int slow, const float (&x)[kChunk<T>]) {
#pragma unroll
      for (int e = 0; e < kChunk<T>; ++e) tile[slow][fast + e] = x[e];
    });
  } else {
    sweep_tile(src, job.from.s_fast, job.from.s_slow, fast0, slow0, n_fast, n_slow, job.from.pairs,
               [&](int fast, int slow, float x0, float x1) {
                 tile[slow][fast] = x0;
                 tile[slow][fast + 1] = x1;
               });
  }
  __syncthreads();
  // pitches are multiples of 64, so what of eight elements lies past the depth lands in the padding
  const int eight = threadIdx.x % 8 * 8;
  if (along.h && fast0 + eight < n_fast) {
    for (int s = threadIdx.x / 8; s < kTile && slow0 + s < n_slow; s += kThreads / 8)
      write_eight(along, fast0 + eight + (slow0 + s) * along.ld, [&](int e) { return tile[s][eight + e] * up_along[s]; });
  }
  if (across.h && slow0 + eight < n_slow) {
    for (int f = threadIdx.x / 8; f < kTile && fast0 + f < n_fast; f += kThreads / 8)
      write_eight(across, slow0 + eight + (fast0 + f) * across.ld, [&](int e) { return tile[eight + e][f] * up_across[f]; });
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

// One matrix with its axes told apart.
struct Oriented {
  Source from;
  HalfTarget along, across;
  SplitTarget mixed_along, mixed_across;
  const RangeGuard* guard;
  int tiles_slow() const { return (from.n_slow + kTile - 1) / kTile; }
  int helper_rows() const { return guard->wide ? (148 + from.tiles_fast - 1) / from.tiles_fast : 0; }
};

void check_job(const PlanesJob& job) {
  for (const HalfTarget* t : {&job.plain, &job.turned}) {
    if (t->h && (!t->largest || t->ld % 64 != 0 || t->ld < (t == &job.plain ? job.rows : job.cols) ||
                 (reinterpret_cast<uintptr_t>(t->h) & 15) != 0 || (reinterpret_cast<uintptr_t>(t->l) & 15) != 0))
      throw std::invalid_argument("half_planes: planes need 16-byte alignment and a pitch that is a multiple of 64");
    if (job.guard.wide && !t->largest)
      throw std::invalid_argument("half_planes: a decision on the range needs the maxima of both orientations");
  }
  if (job.source_type != 0 && job.source_type != 1) throw std::invalid_argument("half_planes: unknown source type");
}

template <typename T>
Oriented oriented(const PlanesJob& job) {
  const bool rows_fast = fast_is_first(job.s_i, job.s_j, job.rows, job.cols);
  Oriented o{};
  o.from.src = job.src;
  o.from.s_fast = rows_fast ? job.s_i : job.s_j;
  o.from.s_slow = rows_fast ? job.s_j : job.s_i;
  o.from.n_fast = rows_fast ? job.rows : job.cols;
  o.from.n_slow = rows_fast ? job.cols : job.rows;
  o.from.tiles_fast = (o.from.n_fast + kTile - 1) / kTile;
  o.from.chunks = reads_chunks(static_cast<const T*>(job.src), o.from.s_fast, o.from.s_slow, o.from.n_slow);
  o.from.pairs = reads_pairs(static_cast<const T*>(job.src), o.from.s_fast, o.from.s_slow, o.from.n_slow);
  o.along = rows_fast ? job.plain : job.turned;
  o.across = rows_fast ? job.turned : job.plain;
  (rows_fast ? o.mixed_along : o.mixed_across) = job.guard.mixed;
  o.guard = &job.guard;
  if (o.tiles_slow() + o.helper_rows() > 65535) throw std::invalid_argument("half_planes: matrix too long");
  return o;
}

template <typename T, bool DECIDED, int N>
void launch(const Oriented* jobs, int count, cudaStream_t stream) {
  ClearGroup<N> clear{};
  LargestGroup<N> largest;
  PlaneGroup<DECIDED, N> planes;
  int longest = 1;
  for (int i = 0; i < count; ++i) {
    const Oriented& o = jobs[i];
    const Source& from = o.from;
    const int tiles = from.tiles_fast * o.tiles_slow();
    clear.words[2 * i] = o.along.largest;
    clear.counts[2 * i] = o.along.largest ? from.n_slow : 0;
    clear.words[2 * i + 1] = o.across.largest;
    clear.counts[2 * i + 1] = o.across.largest ? from.n_fast : 0;
    longest = std::max({longest, from.n_slow, from.n_fast});
    // enough CTAs for every SM several times over before a CTA takes more than one tile
    const int strip = std::clamp(tiles / (148 * 8), 1, 16);
    largest.jobs[i] = LargestJob{from, strip, o.across.largest, o.along.largest};
    largest.blocks.add(from.tiles_fast * ((o.tiles_slow() + strip - 1) / strip));
    PlaneJob<DECIDED>& job = planes.jobs[i];
    job.from = from;
    job.along = o.along;
    job.across = o.across;
    if constexpr (DECIDED) {
      const RangeGuard& guard = *o.guard;
      job.work = MixedWork{guard.wide, {o.along.largest, o.across.largest}, {from.n_slow, from.n_fast}, guard.nearest, o.helper_rows(),
                           mixed_job(static_cast<const T*>(from.src), from.s_fast, from.s_slow, from.n_fast, from.n_slow, o.mixed_along,
                                     o.mixed_across),
                           {basis_job(guard.bases[0]), basis_job(guard.bases[1])}};
    }
    planes.blocks.add(tiles + o.helper_rows() * from.tiles_fast);
  }
  const dim3 block(kThreads);
  check(launch_dependent(clear_kernel<N>, dim3(std::min(8, (longest + kThreads - 1) / kThreads), 2 * count), block, 0, stream, clear),
        "clear_kernel");
  check(launch_dependent(largest_kernel<T, N>, dim3(largest.blocks.total()), block, 0, stream, largest), "largest_kernel");
  check(launch_dependent(half_planes_kernel<T, DECIDED, N>, dim3(planes.blocks.total()), block, 0, stream, planes),
        "half_planes_kernel");
}

}  // namespace

void half_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const HalfTarget& plain,
                 const HalfTarget& turned, const RangeGuard& guard, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || (!plain.h && !turned.h)) return;
  const PlanesJob job{src, source_type, s_i, s_j, rows, cols, plain, turned, guard};
  check_job(job);
  auto go = [&](auto* typed) {
    using T = std::remove_pointer_t<decltype(typed)>;
    const Oriented o = oriented<T>(job);
    if (guard.wide) launch<T, true, 1>(&o, 1, stream);
    else launch<T, false, 1>(&o, 1, stream);
  };
  if (source_type == 0) go(static_cast<float*>(nullptr));
  else go(static_cast<__nv_bfloat16*>(nullptr));
}

void half_planes_group(const PlanesJob* jobs, int count, cudaStream_t stream) {
  if (count < 1 || count > kHalfGroup) throw std::invalid_argument("half_planes: too many matrices for one launch");
  Oriented of_floats[kHalfGroup], of_halves[kHalfGroup];
  int floats = 0, halves = 0;
  for (int i = 0; i < count; ++i) {
    check_job(jobs[i]);
    if (jobs[i].rows <= 0 || jobs[i].cols <= 0 || !jobs[i].guard.wide)
      throw std::invalid_argument("half_planes: matrices of one launch are not empty and have a decision on their range");
    if (jobs[i].source_type == 0) of_floats[floats++] = oriented<float>(jobs[i]);
    else of_halves[halves++] = oriented<__nv_bfloat16>(jobs[i]);
  }
  if (floats) launch<float, true, kHalfGroup>(of_floats, floats, stream);
  if (halves) launch<__nv_bfloat16, true, kHalfGroup>(of_halves, halves, stream);
}

}  // namespace soapb200
