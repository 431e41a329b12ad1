// Host-side interface of the memory-bound kernels (elementwise.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace soapb200 {

// m <- b1 m + (1-b1) g;  v <- b2 v + (1-b2) g^2;  u = (m*inv_bc1) / (sqrt(v)*inv_sqrt_bc2 + eps).
// All four matrices are rows x cols, column-major, with their own pitches.
void adam_update(const float* g, int64_t ldg, float* m, int64_t ldm, float* v, int64_t ldv, float* u, int64_t ldu,
                 int rows, int cols, float beta1, float beta2, float eps, float inv_bc1, float inv_sqrt_bc2,
                 cudaStream_t stream);

// Where one orientation of a matrix goes as operand planes (hi == null: not wanted): column-major with pitch ldo; with `hl`
// (the interleaved bf16 plane of gemm.h, pitch ld16 elements) the low part goes there and `lo` is not written.
struct SplitTarget {
  float* hi = nullptr;
  float* lo = nullptr;
  int64_t ldo = 0;
  uint16_t* hl = nullptr;
  int64_t ld16 = 0;
};

// Operand planes of scale * src[i*s_i + j*s_j], i < rows, j < cols: `plain` the matrix itself (depth rows), `turned` its
// transpose (depth cols).  source_type 0: fp32, 1: bf16.
void split_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const SplitTarget& plain,
                  const SplitTarget& turned, float scale, int nearest, cudaStream_t stream);

// Parameter updates in one pass, contiguous arrays of n elements; parameter (and `gradient`) type 0: fp32, 1: bf16.
//   apply_updates: p <- p * keep (rounded to p's type; skipped for keep == 1), then p <- p - lr * update, the update rounded
//                  to p's type first -- value for value what p.mul_(keep); p.add_(update.to(p.dtype), alpha=-lr) computes.
//   adamw_update:  m <- m + (1 - b1)(g - m), v <- b2 v + (1 - b2) g^2, then the same with (m / bias1) / (sqrt(v / bias2) + eps).
struct UpdateJob {
  void* p;
  const float* update;
  int64_t n;
};
int apply_updates(const UpdateJob* jobs, int count, int type, float keep, float lr, cudaStream_t stream);
void adamw_update(void* p, int type, const void* gradient, float* m, float* v, int64_t n, float beta1_rest, float beta2,
                  float beta2_rest, float bias1, float bias2, float eps, float keep, float lr, cudaStream_t stream);

// out[j] = sum_i a[i, j] * b[i, j] for column-major a, b (deterministic tree reduction per column).
void column_dot(const float* a, int64_t lda, const float* b, int64_t ldb, float* out, int rows, int cols,
                cudaStream_t stream);

// order = stable descending argsort of estimates[j] = sum_{r < parts} table[r + j * ld], j < n <= kOrderMaxLength
// (one CTA, shared-memory bitonic sort; NaN estimates sort last).
constexpr int kOrderMaxLength = 16384;
void order_by_estimate(const float* table, int64_t ld, int parts, int n, int64_t* order, cudaStream_t stream);

// dst(i, j) = src(row_map[i], col_map[j]); a null map is the identity.
void gather2d(const float* src, int64_t s_i, int64_t s_j, float* dst, int64_t d_i, int64_t d_j, const int64_t* row_map,
              const int64_t* col_map, int rows, int cols, cudaStream_t stream);

}  // namespace soapb200
