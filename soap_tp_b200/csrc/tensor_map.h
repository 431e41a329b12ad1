// Tensor maps of K-contiguous operand planes (driver entry point fetched at run time, so no link-time libcuda).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

namespace soapb200 {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult query;
    cudaError_t err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &query);
    if (err != cudaSuccess || query != cudaDriverEntryPointSuccess || ptr == nullptr)
      throw std::runtime_error("cuTensorMapEncodeTiled is not available from the CUDA driver");
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// [rows][depth] elements with `pitch_bytes` between rows; boxes of box_depth x box_rows, zeros beyond the matrix.
inline CUtensorMap encode_k_major(CUtensorMapDataType type, const void* base, int64_t depth, int64_t rows, int64_t pitch_bytes,
                                  int box_depth, int box_rows, CUtensorMapSwizzle swizzle) {
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) throw std::invalid_argument("operand plane must be 16-byte aligned");
  if (pitch_bytes % 16 != 0) throw std::invalid_argument("operand plane pitch must be a multiple of 16 bytes");
  CUtensorMap map;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(depth), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(pitch_bytes)};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_depth), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t elem[2] = {1, 1};
  CUresult res = encode_tiled_fn()(&map, type, 2, const_cast<void*>(base), dims, strides, box, elem,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed with code " + std::to_string(res));
  return map;
}

// The interleaved bf16 plane of a mixed operand (gemm.h): 64 elements (128 bytes) per 32 of K.
inline CUtensorMap encode_interleaved(const uint16_t* base, int64_t K, int64_t rows, int64_t ld, int box_elements, int box_rows) {
  const int64_t extent = 64 * ((K + 31) / 32);
  if (ld % 64 != 0 || ld < extent)
    throw std::invalid_argument("bf16 operand plane pitch must be a multiple of 64 elements covering K");
  return encode_k_major(CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, extent, rows, 2 * ld, box_elements, box_rows,
                        CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace soapb200
