// Tensor maps for TMA, through the runtime's driver entry point lookup (no link against libcuda).
#pragma once

#include <cuda.h>

#include <atomic>

#include "common.cuh"

namespace b200 {

// 2-D tensor [rows][cols] with `row_bytes` between rows, boxes of box_rows x box_cols, out-of-range elements read as zero.
inline int make_map_2d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t cols, uint64_t rows, uint64_t row_bytes,
                       uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static std::atomic<EncodeTiledFn> encode{nullptr};
    EncodeTiledFn fn = encode.load(std::memory_order_acquire);
    if (fn == nullptr) {
        void* q = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &res) != cudaSuccess || q == nullptr) {
            (void)check_launch();
            return B200_ECUDA;
        }
        fn = reinterpret_cast<EncodeTiledFn>(q);
        encode.store(fn, std::memory_order_release);
    }
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = (int)r;
        return B200_ECUDA;
    }
    return B200_OK;
}

}  // namespace b200
