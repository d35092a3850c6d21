// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link-time dependency on the driver).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

typedef CUresult (*lc_encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                       const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// NULL where the driver has no such entry point
inline lc_encode_tiled_fn lc_encode_tiled() {
    static lc_encode_tiled_fn fn = []() -> lc_encode_tiled_fn {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<lc_encode_tiled_fn>(ptr);
    }();
    return fn;
}
// Rows of `row_bytes` (a multiple of 16, base 16-byte aligned) of a matrix, as boxes of `box_rows` rows that are 16 bytes wider than the matrix and
// end each row with zeros.  False where there is no such map (`refused`, no entry point or an error): the caller copies the rows without it.
inline bool lc_wider_rows_map(CUtensorMap *map, bool refused, const void *base, size_t row_bytes, uint32_t rows, uint32_t box_rows) {
    const lc_encode_tiled_fn encode = refused ? nullptr : lc_encode_tiled();
    if (!encode) return false;
    const cuuint64_t dims[2] = {row_bytes / 8, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)(row_bytes + 16) / 8, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
