// Host-side construction of TMA tensor maps (CUtensorMap) for row-major arrays: 2-D, and 3-D as column parts.
// cuTensorMapEncodeTiled lives in the driver library; it is looked up through the runtime
// (cudaGetDriverEntryPoint), so the shared library keeps no link-time dependency on libcuda.
#ifndef SPARSETIR_B200_TMAP_H_
#define SPARSETIR_B200_TMAP_H_

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"

namespace sptir {

// Encodes a map of `rank` dimensions: dims and box in elements, strides (of all but the first dimension) in bytes, multiples of 16;
// the box row (box[0] * element size) must equal the swizzle width for the swizzled modes.  Returns 0, or -1 with the
// error message set.
inline int make_tmap(CUtensorMap* map, CUtensorMapDataType dtype, const void* base, int rank, const cuuint64_t* dims,
                     const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
  using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                CUtensorMapFloatOOBfill);
  static EncodeFn encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<EncodeFn>(fn);
  }();
  if (!encode) return fail("cuTensorMapEncodeTiled is not available from this driver");
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult rc = encode(map, dtype, static_cast<cuuint32_t>(rank), const_cast<void*>(base), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code %d", static_cast<int>(rc));
  return 0;
}

// `rows` x `cols` elements in boxes of `box_rows` x `box_cols`.
inline int make_tmap_2d(CUtensorMap* map, CUtensorMapDataType dtype, const void* base,
                        uint64_t cols, uint64_t rows, uint64_t row_stride_bytes, uint32_t box_cols,
                        uint32_t box_rows, CUtensorMapSwizzle swizzle) {
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {box_cols, box_rows};
  return make_tmap(map, dtype, base, 2, dims, strides, box, swizzle);
}

// The same array as `cols` / `part` column parts: one load brings `box_rows` rows of `box_parts` neighbouring parts, part by part.
inline int make_tmap_parts(CUtensorMap* map, CUtensorMapDataType dtype, const void* base, uint64_t cols, uint64_t rows,
                           uint64_t row_stride_bytes, uint32_t part, uint32_t part_bytes, uint32_t box_rows, uint32_t box_parts,
                           CUtensorMapSwizzle swizzle) {
  const cuuint64_t dims[3] = {part, rows, cols / part};
  const cuuint64_t strides[2] = {row_stride_bytes, part_bytes};
  const cuuint32_t box[3] = {part, box_rows, box_parts};
  return make_tmap(map, dtype, base, 3, dims, strides, box, swizzle);
}

}  // namespace sptir
#endif  // SPARSETIR_B200_TMAP_H_
