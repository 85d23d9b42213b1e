// The driver's encoder of tensor maps, looked up once per process (null: the driver has none).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace brrr {

typedef CUresult (*tmap_encode_t)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline tmap_encode_t tmap_encode() {
    static const tmap_encode_t encode = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) f = nullptr;
        return (tmap_encode_t)f;
    }();
    return encode;
}

}  // namespace brrr
