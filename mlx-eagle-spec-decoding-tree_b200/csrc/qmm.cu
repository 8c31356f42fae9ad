// Entry points of the batched 4-bit affine quantised matmul on row-major (MLX layout) weights:
//
//   y[M,N] = x[M,K] . dequant(W[N,K])^T        W packed 8 x 4 bit per uint32 (element j in bits 4j..4j+3), one fp16 scale and
//                                               bias per 64 k
//
// The kernel is csrc/qmm_gemm.cu.  (Up to 32 rows ran on mma.sync from registers before: 16 x 4096 x 14336 took 46 us there and
// takes 18 us here, one row of 896 x 896 6.3 against 4.2 us; no size was left where it was ahead.)
#include "decode.cuh"
#include "qmm_common.cuh"
#include "qmm_gemm.cuh"

namespace b200 {
namespace {

// Scratch of the allocation-free entry point: lives in the library image, one copy per GPU that
// loads the library, held until the process exits.
constexpr size_t kStaticScratchBytes = 4u << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
constexpr int kMaxDevices = 64;
void* g_static_scratch_ptr[kMaxDevices] = {};

// Device address of the static scratch on the CURRENT device.  The array's name is only a host-side
// handle; the address a kernel may use has to be asked from the runtime, once per device.
int static_scratch_address(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return B200_ECUDA;
    }
    if (dev < 0 || dev >= kMaxDevices) return B200_EINVAL;
    if (g_static_scratch_ptr[dev] == nullptr) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || ptr == nullptr) {
            g_last_cuda_error = (int)e;
            return B200_ECUDA;
        }
        g_static_scratch_ptr[dev] = ptr;
    }
    *out = g_static_scratch_ptr[dev];
    return B200_OK;
}

// Scratch these entry points ask for up to 32 rows, and by which the allocation-free one refuses: partial products of a split along
// K that fills the GPU twice over with 64- or 128-row tiles, two matrices of them for the gate / up pair.  It is the split of a kernel
// that is gone; the rule stays because callers' buffers and refusals follow it.  The split in use fits itself to the room it gets
// (32 x 3584 x 18944 would take 2.3 MiB of these 5.3).
size_t scratch_bytes(int M, int N, int K, bool dual) {
    const int mt = (M + 7) / 8, rw = (dual || mt < 3) ? 16 : 32, target = 2 * gemm_sms(), nchunks = K / kChunkK;
    const int wn = (N + 8 * rw - 1) / (8 * rw) >= target ? 8 : 4;
    const int rows = wn * rw, tiles = (N + rows - 1) / rows;
    if (tiles >= target || tiles > kMaxCounters) return 0;
    int splits = (target + tiles - 1) / tiles;
    splits = splits < (nchunks + 3) / 4 ? splits : (nchunks + 3) / 4;
    const int cps = (nchunks + splits - 1) / splits;
    splits = (nchunks + cps - 1) / cps;
    return splits > 1 ? kCounterBytes + (size_t)splits * tiles * mt * 8 * (dual ? 2 : 1) * rows * sizeof(float) : 0;
}

int qmm_launch(const void* x, const uint32_t* wq, const void* scales, const void* biases, const uint32_t* wq2, const void* scales2,
               const void* biases2, const void* bias, const void* extra, void* y, int M, int N, int K, int group_size, int dtype,
               int epilogue, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
    if (dtype != B200_DTYPE_F16 || group_size != 64) return B200_EUNSUPPORTED;
    if (M < 1 || N < 8 || (N % 8) != 0 || K < kChunkK || (K % kChunkK) != 0) return B200_EINVAL;
    if (epilogue < B200_EPI_NONE || epilogue > B200_EPI_SILU_MUL) return B200_EINVAL;
    const bool dual = epilogue == B200_EPI_SILU_MUL;
    if (!x || !wq || !scales || !biases || !y) return B200_EINVAL;
    if (dual && (!wq2 || !scales2 || !biases2 || bias)) return B200_EINVAL;
    if (epilogue == B200_EPI_RESIDUAL && !extra) return B200_EINVAL;
    if (!aligned16(x) || !aligned16(wq) || !aligned16(y) || !aligned16(bias) || !aligned16(extra) || !aligned16(wq2) || !aligned16(workspace))
        return B200_EALIGN;
    GemmArgs a{};
    a.x = x; a.bias = bias; a.extra = extra; a.y = y;
    a.wq[0] = wq; a.scales[0] = scales; a.biases[0] = biases;
    a.wq[1] = wq2; a.scales[1] = scales2; a.biases[1] = biases2;
    a.M = M; a.N = N; a.K = K; a.epilogue = epilogue;
    gemm_workspace(a, workspace, workspace_bytes);
    if (epilogue == B200_EPI_NONE && a.err != nullptr && chain_matmul_wins(M, N, K, true) &&
        ((reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(biases)) & 3) == 0)
        return chain_matmul({x, wq, scales, biases, bias, y, M, N, K, a.err}, stream);
    // (up to 32 rows no more than the built-in scratch holds, so that the allocation-free call cuts K the same way)
    if (M <= 32 && a.partial_bytes > kStaticScratchBytes - kCounterBytes) a.partial_bytes = kStaticScratchBytes - kCounterBytes;
    return qmm_gemm(a, stream);
}

}  // namespace
}  // namespace b200

extern "C" {

size_t b200_qmm_workspace_bytes(int M, int N, int K) {
    if (M < 1 || N < 8 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return 0;
    if (M > 32) {
        const size_t part = b200::qmm_gemm_partial_bytes(M, N, K, false);
        return part ? b200::kCounterBytes + part : 0;
    }
    const size_t one = b200::scratch_bytes(M, N, K, false), two = b200::scratch_bytes(M, N, K, true);
    return one > two ? one : two;
}

int b200_qmm(const void* x, const uint32_t* wq, const void* scales, const void* biases,
             const void* bias, void* y, int M, int N, int K, int group_size, int dtype,
             void* workspace, size_t workspace_bytes, void* stream) {
    return b200::qmm_launch(x, wq, scales, biases, nullptr, nullptr, nullptr, bias, nullptr, y, M, N, K, group_size, dtype,
                            B200_EPI_NONE, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int b200_qmm_fused(const void* x, const uint32_t* wq, const void* scales, const void* biases,
                   const uint32_t* wq2, const void* scales2, const void* biases2,
                   const void* bias, const void* extra, void* y, int M, int N, int K,
                   int group_size, int dtype, int epilogue,
                   void* workspace, size_t workspace_bytes, void* stream) {
    if (M > 32) return B200_EINVAL;
    return b200::qmm_launch(x, wq, scales, biases, wq2, scales2, biases2, bias, extra, y, M, N, K,
                            group_size, dtype, epilogue, workspace, workspace_bytes,
                            static_cast<cudaStream_t>(stream));
}

size_t b200_qmm_noalloc_max_scratch_bytes(void) { return b200::kStaticScratchBytes; }

int b200_qmm_noalloc(const void* x, const uint32_t* wq, const void* scales, const void* biases,
                     const void* bias, void* y, int M, int N, int K, int group_size, int dtype, void* stream) {
    if (M < 1 || M > 32) return B200_EINVAL;
    // (Only the plain epilogue runs here, so only its scratch counts, not the gate/up pair's.)
    if (N < 8 || K < b200::kChunkK || (K % b200::kChunkK) != 0) return B200_EINVAL;
    if (b200::scratch_bytes(M, N, K, false) > b200::kStaticScratchBytes) return B200_ELIMIT;
    void* scratch = nullptr;
    int rc = b200::static_scratch_address(&scratch);
    if (rc != B200_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // The array keeps whatever the previous call left; the tile counters at its head must start at zero.
    cudaError_t e = cudaMemsetAsync(scratch, 0, b200::kCounterBytes, st);
    if (e != cudaSuccess) {
        b200::g_last_cuda_error = (int)e;
        return B200_ECUDA;
    }
    return b200::qmm_launch(x, wq, scales, biases, nullptr, nullptr, nullptr, bias, nullptr, y, M, N, K,
                            group_size, dtype, B200_EPI_NONE, scratch, b200::kStaticScratchBytes, st);
}

}  // extern "C"
