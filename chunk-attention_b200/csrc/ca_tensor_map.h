// The driver's tensor map encoder, looked up once: the library is not linked against the driver.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace ca {

using TensorMapEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                     const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline TensorMapEncode tensor_map_encoder() {
    static TensorMapEncode fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<TensorMapEncode>(f);
    }();
    return fn;
}

}  // namespace ca
