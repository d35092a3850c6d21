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
