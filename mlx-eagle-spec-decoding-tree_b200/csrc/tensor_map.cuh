// Tensor maps for TMA, through the runtime's driver entry point lookup (no link against libcuda).
#pragma once

#include <cuda.h>

#include <atomic>

#include "common.cuh"

namespace b200 {

// Tensor of `rank` dimensions, innermost first, `strides` bytes between steps of all but that; out-of-range elements read as zero.
inline int make_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                    CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
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
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = (int)r;
        return B200_ECUDA;
    }
    return B200_OK;
}

// 2-D tensor [rows][cols] with `row_bytes` between rows, boxes of box_rows x box_cols.
inline int make_map_2d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t cols, uint64_t rows, uint64_t row_bytes,
                       uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    return make_map(map, type, 2, base, dims, strides, box, swizzle, promotion);
}

// 3-D tensor [z][y][x].
inline int make_map_3d(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t x, uint64_t y, uint64_t z, uint64_t y_bytes, uint64_t z_bytes,
                       uint32_t box_x, uint32_t box_y, uint32_t box_z, CUtensorMapSwizzle swizzle, CUtensorMapL2promotion promotion) {
    const cuuint64_t dims[3] = {x, y, z}, strides[2] = {y_bytes, z_bytes};
    const cuuint32_t box[3] = {box_x, box_y, box_z};
    return make_map(map, type, 3, base, dims, strides, box, swizzle, promotion);
}

}  // namespace b200
