// Memory-bound kernels of the SOAP pipeline: fused Adam, the 3xTF32 operand split (optionally
// transposing), column dot products for the eigenvalue estimates, and index-mapped gathers.
#include <algorithm>
#include <stdexcept>
#include <string>
#include <type_traits>

#include <cuda_bf16.h>

#include "elementwise.h"
#include "gemm.h"
#include "launch_util.h"
#include "split_write.cuh"
#include "tile_sweep.cuh"

namespace soapb200 {
namespace {

inline void check_launch(const char* what) {
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(err));
}

// ---- Adam ---------------------------------------------------------------------------------
// One pass over g, m, v (column-major with independent pitches); the reference issues ten elementwise
// launches for the same arithmetic (src/soap_tp/ops/optimizer.py:36-44).
__global__ void adam_kernel(const float* __restrict__ g, int64_t ldg, float* __restrict__ m, int64_t ldm,
                            float* __restrict__ v, int64_t ldv, float* __restrict__ u, int64_t ldu, int rows, int cols,
                            float beta1, float beta2, float eps, float inv_bc1, float inv_sqrt_bc2) {
  const int64_t total = static_cast<int64_t>(rows) * cols;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i % rows);
    const int64_t c = i / rows;
    const float gi = g[r + c * ldg];
    const float mo = fmaf(beta1, m[r + c * ldm], (1.0f - beta1) * gi);
    const float va = fmaf(beta2, v[r + c * ldv], (1.0f - beta2) * gi * gi);
    m[r + c * ldm] = mo;
    v[r + c * ldv] = va;
    u[r + c * ldu] = (mo * inv_bc1) / (sqrtf(va) * inv_sqrt_bc2 + eps);
  }
}

// Same arithmetic, four elements per thread with 16-byte accesses; used when all four matrices are dense
// (pitch == rows) and 16-byte aligned, i.e. one flat array each.
__global__ void adam_flat4_kernel(const float4* __restrict__ g, float4* __restrict__ m, float4* __restrict__ v,
                                  float4* __restrict__ u, int64_t quads, float beta1, float beta2, float eps, float inv_bc1,
                                  float inv_sqrt_bc2) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < quads;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float4 gi = g[i];
    float4 mo = m[i], va = v[i], out;
#define SOAP_ADAM_LANE(c)                                              \
    mo.c = fmaf(beta1, mo.c, (1.0f - beta1) * gi.c);                   \
    va.c = fmaf(beta2, va.c, (1.0f - beta2) * gi.c * gi.c);            \
    out.c = (mo.c * inv_bc1) / (sqrtf(va.c) * inv_sqrt_bc2 + eps);
    SOAP_ADAM_LANE(x) SOAP_ADAM_LANE(y) SOAP_ADAM_LANE(z) SOAP_ADAM_LANE(w)
#undef SOAP_ADAM_LANE
    m[i] = mo;
    v[i] = va;
    u[i] = out;
  }
}

// ---- parameter updates ---------------------------------------------------------------------------
// Bound by memory (p read and written, the update read: 12 bytes an element for fp32, 8 for bf16) or, for the vectors of a
// model, by the launch: one instead of the two to thirteen that the same arithmetic takes as tensor operations (optimizer step
// over a layer of hidden size 512: 1101 -> 947 us; one-sided step of 32064 x 2048 bf16: 3054 -> 2980 us).
__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T>
__device__ __forceinline__ T round_to(float x);
template <>
__device__ __forceinline__ float round_to<float>(float x) { return x; }
template <>
__device__ __forceinline__ __nv_bfloat16 round_to<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// Each operation rounds to the parameter's type, as separate tensor operations do.
template <typename T>
__device__ __forceinline__ T updated(T p, float update, float keep, float lr) {
  const T kept = keep == 1.0f ? p : round_to<T>(__fmul_rn(to_float(p), keep));
  return round_to<T>(fmaf(-lr, to_float(round_to<T>(update)), to_float(kept)));
}

// Several parameters in one launch, so that those of small matrices do not each wait for the one before.
constexpr int kUpdateGroup = 16;
template <int N>
struct UpdateGroup {
  UpdateJob jobs[N];
  int64_t quads[N];              // leading elements that are aligned to be taken four at a time, in fours
  GroupBlocks<N> blocks;
};

// 16 bytes of update per thread and step where everything is aligned; the rest one by one.
template <typename T, int N>
__global__ void __launch_bounds__(256) apply_updates_kernel(const __grid_constant__ UpdateGroup<N> group, float keep, float lr) {
  struct alignas(4 * sizeof(T)) Four {
    T x[4];
  };
  const int member = group.blocks.member(blockIdx.x), block = blockIdx.x - group.blocks.first(member);
  T* __restrict__ p = static_cast<T*>(group.jobs[member].p);
  const float* __restrict__ update = group.jobs[member].update;
  const int64_t n = group.jobs[member].n, quads = group.quads[member];
  const int64_t first = block * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(group.blocks.count(member)) * blockDim.x;
  for (int64_t i = first; i < quads; i += stride) {
    Four mine = reinterpret_cast<Four*>(p)[i];
    const float4 u = reinterpret_cast<const float4*>(update)[i];
    mine.x[0] = updated(mine.x[0], u.x, keep, lr);
    mine.x[1] = updated(mine.x[1], u.y, keep, lr);
    mine.x[2] = updated(mine.x[2], u.z, keep, lr);
    mine.x[3] = updated(mine.x[3], u.w, keep, lr);
    reinterpret_cast<Four*>(p)[i] = mine;
  }
  for (int64_t i = 4 * quads + first; i < n; i += stride) p[i] = updated(p[i], update[i], keep, lr);
}

template <typename T>
__global__ void __launch_bounds__(256) adamw_kernel(T* __restrict__ p, const T* __restrict__ gradient, float* __restrict__ m,
                                                   float* __restrict__ v, int64_t n, float beta1_rest, float beta2,
                                                   float beta2_rest, float bias1, float bias2, float eps, float keep, float lr) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float g = to_float(gradient[i]);
    // from the nearer end, as lerp does: with a small beta1 an old average far above the gradient must not swallow it
    const float mo = beta1_rest < 0.5f ? fmaf(beta1_rest, g - m[i], m[i]) : fmaf(-(g - m[i]), 1.0f - beta1_rest, g);
    const float va = fmaf(beta2_rest * g, g, __fmul_rn(beta2, v[i]));
    m[i] = mo;
    v[i] = va;
    p[i] = updated(p[i], (mo / bias1) / (sqrtf(va / bias2) + eps), keep, lr);
  }
}

// ---- operand split --------------------------------------------------------------------------
// Bound by memory: the source is read once for both orientations, 64 x 64 tiles turned in shared memory, 8-byte accesses
// along the source's unit stride and along each plane's depth.  32 x 32 tiles with 4-byte accesses took 231 us an orientation
// of an 8192 x 8192 matrix (3.5 TB/s); a one-sided step of 32064 x 2048 bf16 went from 3233 to 3054 us with this kernel.
// `along`: depth runs along the source's fast axis; `across`: along its slow axis.
template <typename T>
__global__ void __launch_bounds__(sweep::kThreads) split_planes_kernel(const T* __restrict__ src, int64_t s_fast, int64_t s_slow,
                                                                      int n_fast, int n_slow, bool pairs, const SplitTarget along,
                                                                      bool along_pairs, const SplitTarget across, bool across_pairs,
                                                                      float scale, int nearest) {
  constexpr int kTile = sweep::kTile;
  __shared__ float tile[kTile][kTile + 1];           // [slow][fast]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fast0 = blockIdx.x * kTile, slow0 = blockIdx.y * kTile;
  sweep::sweep_tile(src, s_fast, s_slow, fast0, slow0, n_fast, n_slow, pairs, [&](int fast, int slow, float x0, float x1) {
    tile[slow][fast] = x0 * scale;
    tile[slow][fast + 1] = x1 * scale;
  });
  __syncthreads();
  if (along.hi && fast0 + 2 * lane < n_fast)
    for (int s = warp; s < kTile && slow0 + s < n_slow; s += 8)
      write_split(along, along_pairs, fast0 + 2 * lane, slow0 + s, n_fast, tile[s][2 * lane], tile[s][2 * lane + 1], nearest);
  if (across.hi && slow0 + 2 * lane < n_slow)
    for (int f = warp; f < kTile && fast0 + f < n_fast; f += 8)
      write_split(across, across_pairs, slow0 + 2 * lane, fast0 + f, n_slow, tile[2 * lane][f], tile[2 * lane + 1][f], nearest);
}

// ---- column dots: out[j] = sum_i a[i, j] * b[i, j] -----------------------------------------
__global__ void __launch_bounds__(256) column_dot_kernel(const float* __restrict__ a, int64_t lda,
                                                         const float* __restrict__ b, int64_t ldb,
                                                         float* __restrict__ out, int rows, int cols) {
  const int j = blockIdx.x;
  if (j >= cols) return;
  float acc = 0.f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) acc = fmaf(a[i + j * lda], b[i + j * ldb], acc);
  __shared__ float partial[256];
  partial[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) partial[threadIdx.x] += partial[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[j] = partial[0];
}

// ---- stable descending order of column sums ------------------------------------------------------
// estimates[j] = sum_r table[r + j * ld] (r < parts, fixed order); order = indices sorted by descending estimate, ties by
// ascending index (what a stable descending argsort returns).  One CTA, bitonic sort of (value, index) pairs in shared
// memory; `padded` is the power of two >= n that the launch was sized for.
__global__ void __launch_bounds__(1024) order_by_estimate_kernel(const float* __restrict__ table, int64_t ld, int parts,
                                                                 int n, int padded, int64_t* __restrict__ order) {
  extern __shared__ unsigned char sort_raw[];
  float* keys = reinterpret_cast<float*>(sort_raw);
  int* index = reinterpret_cast<int*>(keys + padded);
  for (int j = threadIdx.x; j < padded; j += blockDim.x) {
    float total = -INFINITY;                       // padding sorts to the end
    if (j < n) {
      total = 0.f;
      for (int r = 0; r < parts; ++r) total += table[r + j * ld];
      if (total != total) total = -INFINITY;       // a NaN estimate goes last instead of poisoning the network
    }
    keys[j] = total;
    index[j] = j;
  }
  __syncthreads();
  // "a precedes b" in the wanted order: larger value first, smaller index first among equals
  auto precedes = [](float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); };
  for (int size = 2; size <= padded; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < padded / 2; t += blockDim.x) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool ascending_block = (lo & size) == 0;        // blocks alternate direction
        const float va = keys[lo], vb = keys[hi];
        const int ia = index[lo], ib = index[hi];
        const bool in_order = precedes(va, ia, vb, ib);
        if (in_order != ascending_block) {
          keys[lo] = vb; keys[hi] = va;
          index[lo] = ib; index[hi] = ia;
        }
      }
      __syncthreads();
    }
  }
  for (int j = threadIdx.x; j < n; j += blockDim.x) order[j] = index[j];
}

// ---- gather: dst(i, j) = src(row_map[i], col_map[j]) with null maps meaning identity ----------
__global__ void gather2d_kernel(const float* __restrict__ src, int64_t s_i, int64_t s_j, float* __restrict__ dst,
                                int64_t d_i, int64_t d_j, const int64_t* __restrict__ row_map,
                                const int64_t* __restrict__ col_map, int rows, int cols) {
  const int64_t total = static_cast<int64_t>(rows) * cols;
  for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(t % rows);
    const int j = static_cast<int>(t / rows);
    const int64_t si = row_map ? row_map[i] : i;
    const int64_t sj = col_map ? col_map[j] : j;
    dst[i * d_i + j * d_j] = src[si * s_i + sj * s_j];
  }
}

inline int grid_for(int64_t total, int threads) {
  int64_t blocks = (total + threads - 1) / threads;
  const int64_t cap = 148 * 16;
  return static_cast<int>(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace

void adam_update(const float* g, int64_t ldg, float* m, int64_t ldm, float* v, int64_t ldv, float* u, int64_t ldu,
                 int rows, int cols, float beta1, float beta2, float eps, float inv_bc1, float inv_sqrt_bc2,
                 cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return;
  const int64_t total = static_cast<int64_t>(rows) * cols;
  const bool dense = (cols == 1 || (ldg == rows && ldm == rows && ldv == rows && ldu == rows)) && total % 4 == 0;
  const bool aligned = ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                         reinterpret_cast<uintptr_t>(u)) & 15) == 0;
  if (dense && aligned) {
    adam_flat4_kernel<<<grid_for(total / 4, 256), 256, 0, stream>>>(
        reinterpret_cast<const float4*>(g), reinterpret_cast<float4*>(m), reinterpret_cast<float4*>(v),
        reinterpret_cast<float4*>(u), total / 4, beta1, beta2, eps, inv_bc1, inv_sqrt_bc2);
    check_launch("adam_flat4_kernel");
    return;
  }
  adam_kernel<<<grid_for(static_cast<int64_t>(rows) * cols, 256), 256, 0, stream>>>(
      g, ldg, m, ldm, v, ldv, u, ldu, rows, cols, beta1, beta2, eps, inv_bc1, inv_sqrt_bc2);
  check_launch("adam_kernel");
}

namespace {
template <typename T, int N>
void launch_updates(const UpdateJob* jobs, int count, float keep, float lr, cudaStream_t stream) {
  UpdateGroup<N> group;
  for (int i = 0; i < count; ++i) {
    const UpdateJob& job = jobs[i];
    const bool aligned = reinterpret_cast<uintptr_t>(job.p) % (4 * sizeof(T)) == 0 && (reinterpret_cast<uintptr_t>(job.update) & 15) == 0;
    group.jobs[i] = job;
    group.quads[i] = aligned ? job.n / 4 : 0;
    group.blocks.add(grid_for(aligned ? (job.n + 3) / 4 : job.n, 256));
  }
  apply_updates_kernel<T, N><<<group.blocks.total(), 256, 0, stream>>>(group, keep, lr);
  check_launch("apply_updates_kernel");
}
}  // namespace

int apply_updates(const UpdateJob* jobs, int count, int type, float keep, float lr, cudaStream_t stream) {
  if (type != 0 && type != 1) throw std::invalid_argument("apply_updates: unknown parameter type");
  auto go = [&](auto* typed, const UpdateJob* some, int n) {
    using T = std::remove_pointer_t<decltype(typed)>;
    if (n == 1) launch_updates<T, 1>(some, n, keep, lr, stream);
    else launch_updates<T, kUpdateGroup>(some, n, keep, lr, stream);
  };
  const int64_t width = type == 0 ? sizeof(float) : sizeof(__nv_bfloat16);
  auto overlap = [&](const UpdateJob& a, const UpdateJob& b) {
    const auto x = reinterpret_cast<uintptr_t>(a.p), y = reinterpret_cast<uintptr_t>(b.p);
    return x < y + width * b.n && y < x + width * a.n;
  };
  UpdateJob some[kUpdateGroup];
  int n = 0, launches = 0;
  auto flush = [&] {
    if (n == 0) return;
    ++launches;
    if (type == 0) go(static_cast<float*>(nullptr), some, n);
    else go(static_cast<__nv_bfloat16*>(nullptr), some, n);
    n = 0;
  };
  for (int i = 0; i < count; ++i) {
    if (jobs[i].n <= 0) continue;
    // parameters that share memory are updated one after the other
    if (n == kUpdateGroup || std::any_of(some, some + n, [&](const UpdateJob& other) { return overlap(other, jobs[i]); })) flush();
    some[n++] = jobs[i];
  }
  flush();
  return launches;
}

void adamw_update(void* p, int type, const void* gradient, float* m, float* v, int64_t n, float beta1_rest, float beta2,
                  float beta2_rest, float bias1, float bias2, float eps, float keep, float lr, cudaStream_t stream) {
  if (n <= 0) return;
  auto go = [&](auto* typed) {
    using T = std::remove_pointer_t<decltype(typed)>;
    adamw_kernel<T><<<grid_for(n, 256), 256, 0, stream>>>(typed, static_cast<const T*>(gradient), m, v, n, beta1_rest, beta2,
                                                          beta2_rest, bias1, bias2, eps, keep, lr);
    check_launch("adamw_kernel");
  };
  if (type == 0) go(static_cast<float*>(p));
  else if (type == 1) go(static_cast<__nv_bfloat16*>(p));
  else throw std::invalid_argument("adamw_update: unknown parameter type");
}

namespace {
template <typename T>
void launch_split(const T* src, int64_t s_fast, int64_t s_slow, int n_fast, int n_slow, const SplitTarget& along,
                  const SplitTarget& across, float scale, int nearest, cudaStream_t stream) {
  const dim3 grid((n_fast + sweep::kTile - 1) / sweep::kTile, (n_slow + sweep::kTile - 1) / sweep::kTile);
  if (grid.y > 65535) throw std::invalid_argument("split_planes: matrix too long");
  split_planes_kernel<T><<<grid, sweep::kThreads, 0, stream>>>(src, s_fast, s_slow, n_fast, n_slow,
                                                               sweep::reads_pairs(src, s_fast, s_slow, n_slow), along,
                                                               writes_pairs(along), across, writes_pairs(across), scale, nearest);
  check_launch("split_planes_kernel");
}
}  // namespace

void split_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const SplitTarget& plain,
                  const SplitTarget& turned, float scale, int nearest, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || (!plain.hi && !turned.hi)) return;
  const bool rows_fast = cols == 1 || (rows > 1 && s_i <= s_j);       // the axis with the smaller stride is swept by the lanes
  auto go = [&](auto* typed) {
    if (rows_fast) launch_split(typed, s_i, s_j, rows, cols, plain, turned, scale, nearest, stream);
    else launch_split(typed, s_j, s_i, cols, rows, turned, plain, scale, nearest, stream);
  };
  if (source_type == 0) go(static_cast<const float*>(src));
  else if (source_type == 1) go(static_cast<const __nv_bfloat16*>(src));
  else throw std::invalid_argument("split_planes: unknown source type");
}

void column_dot(const float* a, int64_t lda, const float* b, int64_t ldb, float* out, int rows, int cols,
                cudaStream_t stream) {
  if (cols <= 0) return;
  column_dot_kernel<<<cols, 256, 0, stream>>>(a, lda, b, ldb, out, rows, cols);
  check_launch("column_dot_kernel");
}

void order_by_estimate(const float* table, int64_t ld, int parts, int n, int64_t* order, cudaStream_t stream) {
  if (n <= 0) return;
  int padded = 1;
  while (padded < n) padded <<= 1;
  if (padded > kOrderMaxLength) throw std::invalid_argument("order_by_estimate: more entries than one CTA's shared memory sorts");
  const size_t smem = static_cast<size_t>(padded) * (sizeof(float) + sizeof(int));
  static PerDeviceOnce configured;
  allow_dynamic_smem(reinterpret_cast<const void*>(order_by_estimate_kernel), kOrderMaxLength * 8, configured, "order_by_estimate");
  order_by_estimate_kernel<<<1, 1024, smem, stream>>>(table, ld, parts, n, padded, order);
  check_launch("order_by_estimate_kernel");
}

void gather2d(const float* src, int64_t s_i, int64_t s_j, float* dst, int64_t d_i, int64_t d_j, const int64_t* row_map,
              const int64_t* col_map, int rows, int cols, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return;
  gather2d_kernel<<<grid_for(static_cast<int64_t>(rows) * cols, 256), 256, 0, stream>>>(src, s_i, s_j, dst, d_i, d_j,
                                                                                     row_map, col_map, rows, cols);
  check_launch("gather2d_kernel");
}

}  // namespace soapb200
