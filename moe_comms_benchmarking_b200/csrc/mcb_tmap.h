// Host side: tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mcb {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) fn = nullptr;
    return reinterpret_cast<EncodeTiledFn>(fn);
  }();
  return encode;
}

// Each fills `out` (128 bytes, 64-byte aligned host memory).
inline int make_tmap(void* out, CUtensorMapDataType type, uint32_t elem, const void* base, uint64_t rows, uint64_t cols,
                     uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle) {
  if (!encode_tiled()) return (int)cudaErrorNotSupported;
  if (!rows || cols % box_cols || (reinterpret_cast<uintptr_t>(base) & 15)) return (int)cudaErrorInvalidValue;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * elem};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_tiled()(reinterpret_cast<CUtensorMap*>(out), type, 2, const_cast<void*>(base), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}
// A row-major bf16 matrix [rows, cols] in boxes of box_rows x 64 columns with the 128-byte swizzle.
inline int make_tmap_bf16(void* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, rows, cols, box_rows, 64, CU_TENSOR_MAP_SWIZZLE_128B);
}
// `bytes` of contiguous memory as rows of 2 KB, in boxes of box_rows rows, as they lie in memory.
inline int make_tmap_flat(void* out, const void* base, uint64_t bytes, uint32_t box_rows) {
  return make_tmap(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, base, bytes / 2048, 256, box_rows, 256, CU_TENSOR_MAP_SWIZZLE_NONE);
}

}  // namespace mcb
