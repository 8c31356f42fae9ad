// Host interface of the large-M quantised matmul (csrc/qmm_gemm.cu) for the other files of the library.
#pragma once

#include "common.cuh"
#include "qmm_common.cuh"

namespace b200 {

struct GemmArgs {
    const void* x;               // [M][K] fp16, row-major
    const void* w_tiled;         // streaming layout, or NULL: row-major weights below
    const void* w2_tiled;        // up_proj (B200_EPI_SILU_MUL)
    const uint32_t* wq[2];       // row-major packed weights, scales, biases (gate / up)
    const void* scales[2];
    const void* biases[2];
    const void* bias;            // [N] or NULL
    const void* extra;           // residual [M][N] (B200_EPI_RESIDUAL)
    void* y;                     // [M][N]; float with B200_EPI_F32
    int M, N, K;
    int epilogue;
    int* counters;               // 896 tickets of the K split, zero before first use, restored by every launch
    int* err;                    // set when a bounded wait gives up; may be NULL
    void* partial;               // fp32 partial products of the K split
    size_t partial_bytes;        // 0: no split
};

// The library's usual workspace: 4 KiB of counters (the last one the error word), then the partial products.
inline void gemm_workspace(GemmArgs& a, void* workspace, size_t bytes) {
    if (workspace == nullptr || bytes < (size_t)kCounterBytes) return;
    a.counters = static_cast<int*>(workspace);
    a.err = a.counters + kMaxCounters - 1;
    a.partial = static_cast<char*>(workspace) + kCounterBytes;
    a.partial_bytes = bytes - kCounterBytes;
}

// Work split of csrc/qmm_pair.cu: tokens per tile (a multiple of 32, at most 256), 256-row tiles, token tiles, K ranges of cps chunks; its cost
// in cycles.
struct PairPlan {
    int NT, row_items, tok_items, splits, cps;
    double cost;
};
int qmm_pair(const GemmArgs& a, const PairPlan& plan, cudaStream_t stream);

int gemm_sms();                  // SMs of the current device
size_t qmm_gemm_partial_bytes(int M, int N, int K, bool dual);


// y = epilogue(x . dequant(W)^T); every pointer 16-byte aligned, K % 128 == 0, N % 8 == 0, M >= 1.
int qmm_gemm(const GemmArgs& a, cudaStream_t stream);

}  // namespace b200
