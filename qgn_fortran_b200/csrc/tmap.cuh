// tmap.cuh -- tensor maps for the TMA copies (cp.async.bulk.tensor).  The encoder is a driver entry
// point, looked up once, so the library needs no link against the driver.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace qgn {

using TensorMapEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                     const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline TensorMapEncode tensor_map_encoder() {
    static const TensorMapEncode encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &r) != cudaSuccess) f = nullptr;
        return reinterpret_cast<TensorMapEncode>(f);
    }();
    return encode;
}

// a tiled map of `rank` dimensions (innermost first; strides of all but the innermost, in bytes),
// boxes of `box` elements, out-of-range elements read as zero
inline cudaError_t tensor_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base,
                              const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                              CUtensorMapSwizzle swizzle) {
    const TensorMapEncode encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, type, (cuuint32_t)rank, const_cast<void*>(base), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace qgn
