// TMA descriptors: the driver's encoder, and the cached factory of the GEMM kernels (defined in gemm_tcgen05.cu).
#pragma once
#include <cuda.h>
#include <stdint.h>

namespace b200 {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// cuTensorMapEncodeTiled of the driver that is loaded (nullptr: none)
EncodeTiledFn tensor_map_encoder();
// bf16 row-major [rows, cols] (row stride ld elements) -> tiles of box_rows x 64 elements, 128B swizzle
bool gemm_make_tmap(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
// 1-byte elements (e4m3) row-major [rows, cols] -> tiles of box_rows x 128 elements (one 128 B swizzle row)
bool gemm_make_tmap_u8(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
}  // namespace b200
