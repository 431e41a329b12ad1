// Host-side interface of the fp16-pair GEMM (gemm_half.cu) and of the kernels that make its operands (half_planes.cu).
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "elementwise.h"

namespace soapb200 {

// A K x cols operand as scaled fp16 planes: element (k, c) is
//   scale[(k / 128) * scale_stride + c] * (h[k + c * ld] + l[k + c * ld]),
// scales being powers of two that bring the largest magnitude of the vector (scale_stride == 0: the whole K-vector c;
// else: its 128-element block) into [2^14, 2^15).  h = rn_fp16(x), l = rn_fp16(x - h) are off by 2^-23 of an element or by
// 2^-39 of the largest one of its vector or block (fp16's smallest step), whichever is more.  l is null for bf16 values,
// which h holds by itself down to 2^-32 of the largest one.
//
// The second kind of error is hidden by the rounding of an fp32 sum that the largest element is part of -- unless the other
// operand is nearly zero there, as the eigenvectors of a graded matrix are: a coordinate of a rotated gradient that only the
// small rows or columns feed would come out with fewer bits than from the mixed form (gemm.h, 2^-20 of each element), and
// Adam divides it by its own size.  So a rotation decides on the device (RangeGuard) which form its products take.
struct HalfOperand {
  const uint16_t* h;
  const uint16_t* l;
  int64_t ld;              // multiple of 64
  const float* scale;
  int64_t scale_stride;    // 0 for the second operand of a product, whose scales are applied after the sum over K
  // The same operand in the mixed form, read where HalfProblem::wide says so: maps of its two planes (mixed_maps).
  const CUtensorMap* mixed = nullptr;
  // Maps of h and l where they were made with the planes (half_maps); null: made for the product.
  const CUtensorMap* maps = nullptr;
};
// The tensor maps of K x cols planes, fp16 pairs and mixed, which belong to scratch or to a basis's planes and are made once with
// them (a map takes the host 0.2 us, and a step's products need forty).
void half_maps(CUtensorMap (&maps)[2], const uint16_t* h, const uint16_t* l, int64_t ld, int64_t K, int64_t cols);
void mixed_maps(CUtensorMap (&maps)[2], const SplitTarget& planes, int64_t K, int64_t cols);

constexpr int kHalfScaleBlock = 128;

struct HalfProblem {
  int M, N, K;
  int mode;                // kEpiStore, kEpiSplit, kEpiAdam or kEpiRowMajor (gemm.h)
  int symmetric;           // A == B: tiles on and below the diagonal, mirrored (kEpiStore)
  int tiles;               // 0: chosen by size; 1: single CTAs (128 x 128); 2: CTA pairs (256 x 256)
  float alpha, beta;
  float* C;
  int64_t ldc;
  // kEpiSplit, kEpiAdam: the result as an operand of depth M with one scale per 128 rows and column
  uint16_t* Ch;
  uint16_t* Cl;
  int64_t ldp;
  float* Cscale;
  int64_t ldscale;
  float* mom;
  float* var;
  int64_t ldm, ldv;
  float beta1, beta2, eps, inv_bc1, inv_sqrt_bc2;
  // Device word (null: never): where it is set the product runs on the operands' mixed form -- tf32 and two bf16 corrections,
  // drained every 64 of K like gemm_tf32x3 -- and kEpiSplit, kEpiAdam write the mixed form, here.
  const int* wide;
  int settled;             // the word was written before the kernel ahead of this one in the stream began
  SplitTarget mixed;
};

// Whether such a product is large enough for CTA pairs, and whether it runs on them where it does not say (the pair switch may be off).
bool half_fills_pairs(int M, int N, bool symmetric);
bool half_on_pairs(int M, int N, bool symmetric);

void gemm_half(const HalfOperand& a, const HalfOperand& b, const HalfProblem& prob, int* status, cudaStream_t stream);

// Up to kHalfGroup products with the same epilogue in one launch of single CTAs.
constexpr int kHalfGroup = 8;
struct HalfJob {
  HalfOperand a, b;
  HalfProblem problem;
};
void gemm_half_group(const HalfJob* jobs, int count, int* status, cudaStream_t stream);

// Where one orientation of a matrix goes as scaled fp16 planes (h == null: not wanted).  `scale` has one entry per vector,
// `largest` is scratch of the same length (needed without planes too where a RangeGuard looks at it).
struct HalfTarget {
  uint16_t* h;
  uint16_t* l;             // null: one term
  int64_t ld;
  float* scale;
  uint32_t* largest;
};

// A basis that is kept as fp16 planes, and where its mixed form goes on demand.
struct WideBasis {
  const float* src;        // element (i, j) at src[i * s_i + j * s_j], i, j < size
  int64_t s_i, s_j;
  int size;
  SplitTarget plain, turned;
};

// Decides whether scaled fp16 pairs hold a matrix that is to be rotated.  They do unless a row's or a column's largest
// magnitude lies more than kRangeOrders binary orders under the matrix's (all zeros included: what meets such a row is what a
// basis nearly misses), or the matrix has infinities or NaN.
//
// Why the rows and columns of the matrix: Y = Q_L^T G Q_R passes through T = G^T Q_L, whose row j is as long as column j of G.
// The floor of 2^-39 of the largest puts an error of 2^-39 |G|max on a column of Y, whose fp32 rounding is at least 2^-24 of
// the shortest column of G; likewise for rows.  Within 2^12 of each other the floor is 2^-27 of every row and column, and 2^-20,
// what the mixed form keeps, where one entry stands against rows of 16384.
constexpr int kRangeOrders = 12;
struct RangeGuard {
  int* wide;               // device word: set to 1 (too wide) or 0; null: no decision
  SplitTarget mixed;       // `plain` in the mixed form, written where it is set
  WideBasis bases[2];      // likewise
  int nearest;             // rounding of tf32 values, as split_planes
};

// The operand `plain` (depth rows, vectors = columns) and / or `turned` (depth cols, vectors = rows) of src[i*s_i + j*s_j],
// i < rows, j < cols; source_type 0: fp32, 1: bf16.
void half_planes(const void* src, int source_type, int64_t s_i, int64_t s_j, int rows, int cols, const HalfTarget& plain,
                 const HalfTarget& turned, const RangeGuard& guard, cudaStream_t stream);
// The same for up to kHalfGroup matrices in the same launches; all with a decision on the range.
struct PlanesJob {
  const void* src;
  int source_type;
  int64_t s_i, s_j;
  int rows, cols;
  HalfTarget plain, turned;
  RangeGuard guard;
};
void half_planes_group(const PlanesJob* jobs, int count, cudaStream_t stream);

// A matrix to be rotated by two bases (steady_step.cpp).
struct Rotation {
  const void* source;
  int source_type;
  int64_t s_i, s_j;
  int rows, cols;
  HalfTarget x, xt;                                          // planes of G (depth rows) and G^T (depth cols), written
  HalfOperand left, left_turned, right, right_turned;        // planes of Q_L, Q_L^T, Q_R, Q_R^T
  HalfOperand middle;                                        // scratch planes cols x rows, scales per block
  SplitTarget mixed_middle;                                  // the same in the mixed form
  const CUtensorMap* mixed_source;                           // maps of guard.mixed
  const CUtensorMap *x_maps, *xt_maps;                       // of x and xt
  RangeGuard guard;
};

// out = Q_L^T G Q_R, or Q_L G Q_R^T (`turned`), column-major rows x cols; may overwrite the source.
void rotate_half(const Rotation& r, bool turned, float* out, int64_t ldc, int* status, cudaStream_t stream);

// One ordinary step of a rows x cols parameter: every operand, result and scalar of its launches.
struct SteadyStep {
  Rotation rotation;                                         // of the gradient
  HalfOperand update;                                        // scratch planes rows x cols, scales per block
  SplitTarget mixed_update;
  float* momentum;
  int64_t ldm;
  float* variance;
  int64_t ldv;
  float* out;                                                // rows x cols, row-major
  float* left_gram;
  int64_t ld_left;
  float* right_gram;
  int64_t ld_right;
  double beta;
  float beta1, beta2, eps, inv_bc1, inv_sqrt_bc2;
  int phases;                                                // kStep*
  cudaStream_t side;                                         // the averages run here, beside the rotations (or the step's own)
};
constexpr int kStepPlanes = 1, kStepForward = 2, kStepBackward = 4, kStepAverages = 8;
void steady_step(const SteadyStep& s, int* status, cudaStream_t stream);
// Whether no product of such a step is large enough for CTA pairs, whether they are in use or not, so that several small parameters
// can share its launches; and the steps of up to kHalfGroup such parameters (all phases; scratch of their own each).
bool steady_step_shares(int rows, int cols);
// Whether both averages of a step run on single CTAs, and so in one launch.
bool averages_share(int rows, int cols);
void steady_steps(const SteadyStep* steps, int count, int* status, cudaStream_t stream);

// Scale of a vector or block from the bit pattern of its largest magnitude (clamped so that both factors are normal):
// x * multiplier is what the planes hold, `inverse` undoes it.  Infinities and NaN pass through with a factor of one.
struct HalfScale {
  float multiplier, inverse;
};
#ifdef __CUDACC__
__device__ __forceinline__ HalfScale half_scale(uint32_t largest_bits) {
  const uint32_t exponent = largest_bits >> 23;
  if (exponent == 255u) return HalfScale{1.0f, 1.0f};
  const uint32_t up = exponent < 15u ? 253u : 268u - exponent;      // biased exponent of 2^(14 - floor(log2 largest))
  return HalfScale{__uint_as_float(up << 23), __uint_as_float((254u - up) << 23)};
}
#endif

}  // namespace soapb200
