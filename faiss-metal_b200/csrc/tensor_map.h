// cuTensorMapEncodeTiled, which encodes the operands' tensor maps, as the driver exports it.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace b200f {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Looked up once; threads that make their first searches at the same time wait for the one that looks.  Null: no such driver.
inline EncodeTiledFn get_encode_fn() {
    static const EncodeTiledFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(ptr);
        (void)cudaGetLastError();
        return EncodeTiledFn(nullptr);
    }();
    return fn;
}

}  // namespace b200f
