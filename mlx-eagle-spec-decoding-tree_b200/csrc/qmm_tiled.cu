// Streaming ("tiled") weight layout: the one-off re-layout and the entry points of the matmul on it (kernel: csrc/qmm_gemm.cu).
//
// Offline re-layout (the analogue of the reference's swizzle.py / kernels/swizzle.metal): the matrix
// is cut into records of 16 rows x 128 k.  A record is 1152 contiguous bytes: 1024 bytes of packs
// in exactly the order the 32 lanes of a warp consume them (lane (g,t) owns 16 bytes of row g and
// 16 bytes of row g+8: the packs of k-blocks t, 4+t, 8+t, 12+t), then 128 bytes of {scale, bias}
// pairs (row-major, two 64-k groups per row).  Inside a pack the nibbles are re-ordered so that
// the mask pairs 0x000f000f, 0x00f000f0 (and the same after >> 8) yield ADJACENT k pairs
// (k0,k1) (k2,k3) (k4,k5) (k6,k7): the activations can then stay in their natural order.  Records are ordered [64-row block][k chunk][16-row
// tile of the block], so everything a CTA needs for one k chunk of a 64-row block is one
// contiguous 4.5 KiB run, and consecutive chunks follow each other.
#include "decode.cuh"
#include "pipeline.cuh"
#include "qmm_common.cuh"
#include "qmm_gemm.cuh"

namespace b200 {
namespace {

constexpr int kRec = 1152;            // bytes per 16-row x 128-k record
constexpr int kBlockRows = 64;        // rows per layout block (4 records per chunk)

// ---- re-layout -------------------------------------------------------------------------------
__global__ void relayout_kernel(const uint32_t* __restrict__ wq, const __half* __restrict__ scales,
                                const __half* __restrict__ biases, uint32_t* __restrict__ out, int N, int K) {
    const int nchunks = K / kChunkK;
    const int rec = blockIdx.x;                 // (block64 * nchunks + c) * 4 + tile in block
    const int tib = rec & 3, bc = rec >> 2;
    const int blk = bc / nchunks, c = bc - blk * nchunks;
    const int t16 = blk * 4 + tib;
    const int i = threadIdx.x;                  // 0..287: u32 index inside the record
    pdl_wait();
    uint32_t v = 0;
    if (i < 256) {
        const int hh = i >> 7, lane = (i >> 2) & 31, j = i & 3;
        const int row = t16 * 16 + (lane >> 2) + 8 * hh;
        if (row < N) {
            const uint32_t w = wq[(size_t)row * (K / 8) + c * 16 + j * 4 + (lane & 3)];
            // element e (bits 4e..4e+3 in the MLX pack) moves to nibble (e >> 1) + 4 * (e & 1)
#pragma unroll
            for (int e = 0; e < 8; e++) v |= ((w >> (4 * e)) & 0xfu) << (4 * ((e >> 1) + 4 * (e & 1)));
        }
    } else {
        const int q = i - 256, row = t16 * 16 + (q >> 1), grp = q & 1;
        if (row < N) {
            const unsigned short s = __half_as_ushort(scales[(size_t)row * (K / 64) + 2 * c + grp]);
            const unsigned short b = __half_as_ushort(biases[(size_t)row * (K / 64) + 2 * c + grp]);
            v = (uint32_t)s | ((uint32_t)b << 16);
        }
    }
    out[(size_t)rec * (kRec / 4) + i] = v;
}

}  // namespace
}  // namespace b200

extern "C" {

size_t b200_qmm_tiled_bytes(int N, int K) {
    if (N < 1 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return 0;
    return (size_t)((N + b200::kBlockRows - 1) / b200::kBlockRows) * (K / b200::kChunkK) * 4 * b200::kRec;
}

int b200_qmm_relayout(const uint32_t* wq, const void* scales, const void* biases, void* out, int N, int K,
                      void* stream) {
    if (!wq || !scales || !biases || !out || N < 1 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return B200_EINVAL;
    if (!b200::aligned16(out)) return B200_EALIGN;
    const int recs = ((N + b200::kBlockRows - 1) / b200::kBlockRows) * (K / b200::kChunkK) * 4;
    b200::launch_kernel(b200::relayout_kernel, dim3(recs), dim3(b200::kRec / 4), 0, static_cast<cudaStream_t>(stream),
                        wq, static_cast<const __half*>(scales), static_cast<const __half*>(biases),
                        static_cast<uint32_t*>(out), N, K);
    return b200::check_launch();
}

size_t b200_qmm_tiled_workspace_bytes(int M, int N, int K) {
    if (M < 1 || N < 8 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return 0;
    if (M > 32) M = 32;
    const size_t one = b200::qmm_gemm_partial_bytes(M, N, K, false), two = b200::qmm_gemm_partial_bytes(M, N, K, true);
    return b200::kCounterBytes + (one > two ? one : two);
}

int b200_qmm_tiled(const void* x, const void* wt, const void* wt2, const void* bias, const void* extra, void* y,
                   int M, int N, int K, int epilogue, void* workspace, size_t workspace_bytes, void* stream) {
    if (M < 1 || M > 32 || N < 8 || (N % 8) != 0 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return B200_EINVAL;
    if (epilogue < B200_EPI_NONE || epilogue > B200_EPI_F32) return B200_EINVAL;
    if (epilogue == B200_EPI_F32 && bias) return B200_EINVAL;
    const bool dual = epilogue == B200_EPI_SILU_MUL;
    if (!x || !wt || !y || !workspace || (dual && (!wt2 || bias)) || (epilogue == B200_EPI_RESIDUAL && !extra))
        return B200_EINVAL;
    if (!b200::aligned16(x) || !b200::aligned16(wt) || !b200::aligned16(wt2) || !b200::aligned16(y) ||
        !b200::aligned16(bias) || !b200::aligned16(extra) || !b200::aligned16(workspace))
        return B200_EALIGN;
    if (workspace_bytes < (size_t)b200::kCounterBytes) return B200_EWORKSPACE;
    if (epilogue == B200_EPI_NONE && b200::chain_matmul_wins(M, N, K, false))
        return b200::chain_matmul({x, wt, nullptr, nullptr, bias, y, M, N, K, static_cast<int*>(workspace) + b200::kMaxCounters - 1},
                                  static_cast<cudaStream_t>(stream));
    b200::GemmArgs a{};
    a.x = x; a.w_tiled = wt; a.w2_tiled = wt2; a.bias = bias; a.extra = extra; a.y = y;
    a.M = M; a.N = N; a.K = K; a.epilogue = epilogue;
    b200::gemm_workspace(a, workspace, workspace_bytes);
    return b200::qmm_gemm(a, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
