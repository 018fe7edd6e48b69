// Host side of the TMA: cuTensorMapEncodeTiled through the runtime's entry-point query (the library links no libcuda).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace b2 {

inline decltype(&cuTensorMapEncodeTiled) map_encoder() {
    static const auto encode = []() -> decltype(&cuTensorMapEncodeTiled) {
        void * f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(f);
    }();
    return encode;
}
inline bool encode_map(CUtensorMap & m, CUtensorMapDataType type, int rank, const void * base, const cuuint64_t * dims, const cuuint64_t * strides,
                       const cuuint32_t * box, CUtensorMapSwizzle swizzle) {
    const cuuint32_t steps[4] = {1, 1, 1, 1};
    const auto encode = map_encoder();
    return encode && encode(&m, type, rank, const_cast<void *>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace b2
