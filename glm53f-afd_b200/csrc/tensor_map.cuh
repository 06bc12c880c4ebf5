// The tensor-map encoder for the host code of the kernels that copy by tensor maps.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace kda {

// The driver's encoder, looked up once through the runtime (the library does not link libcuda).
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiled encode_tiled() {
    static EncodeTiled fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qr) != cudaSuccess || qr != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiled>(f);
    }();
    return fn;
}

}  // namespace kda
