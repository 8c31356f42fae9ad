// The kernel chain of a forward pass (csrc/decode.cu) as csrc/forward.cu calls it.
#pragma once

#include "common.cuh"

namespace b200 {

// What b200_forward has checked and laid out of the descriptor: everything is valid, tp_world <= 1.
struct ChainArgs {
    const b200_forward_desc* d;
    const void* const* layers;   // host copy of the layer table, or NULL: the kernels read the descriptor's
    int* err;             // error word
    float* ssq;           // [hidden / 32][32]
    float2* cs;           // [32][64]
    int splits[5];        // K split (cluster size) asked for per phase A, C, D, E, head; 0 = planner
};

int forward_chain(const ChainArgs& a, cudaStream_t stream);

// The layers of a prompt pass (embedding to the last layer's h) through the chain's kernels, tiles of 32 tokens side by side.
struct ChainPrompt {
    const b200_prefill_desc* d;  // checked; xn holds h * w_norm
    int* err;
    float* ssq;                  // [hidden / 32][tokens rounded up to 32]
    float2* cs;                  // [tokens][64]
    unsigned long long* mask;    // [tokens], at most 64, and committed length for the attention; or NULL
    int* prefix;
    int (*attention)(const void* context, int row0, cudaStream_t stream);
    const void* context;
};
int chain_prompt(const ChainPrompt& c, cudaStream_t stream);

// y[M][N] = x[M][K] . W^T (+ bias), M <= 32, by the chain's matmul kernel on its own.  W in the streaming layout, or as quantised
// (packs, with 4-byte aligned scales and biases).
struct ChainMatmul {
    const void* x;
    const void* w;
    const void* scales;
    const void* biases;
    const void* bias;
    void* y;
    int M, N, K;
    int* err;
};
// Few chunks per SM: the clusters of this kernel add up K without going through memory and its CTAs are half as large.  (8 rows,
// streaming layout: 1024 x 4096 6.2 -> 3.8 us, 8192 x 2048 7.4 -> 5.3, 19200 x 256 4.0 -> 3.7.)  Beyond ten or so its three groups of
// dequant warps stream less than the four of the large-M kernel (2048 x 18944, 16 chunks: 10.0 against 11.2 us; 4096 x 14336, 24:
// the same; 19200 x 18944: 54 against 77).
// As quantised it has scales to fetch and pairs to reorder: it wins later, up to 16 rows from a few chunks on (8 x 896 x 896 4.9 ->
// 4.1, 8 x 1024 x 4096 7.3 -> 5.6; 8 x 128 x 256 3.0 against 3.4), beyond from about two per SM (31 x 8192 x 2048 8.6 -> 7.8; 31 x
// 4096 x 1024 5.4 against 5.8), and loses earlier (8 x 19200 x 1280, ten per SM: 9.8 against 10.3).
inline bool chain_matmul_wins(int M, int N, int K, bool as_quantised) {
    const long long chunks = (long long)((N + 127) / 128) * (K / 128);
    if (M > 32) return false;
    return as_quantised ? chunks <= 1152 && chunks >= (M <= 16 ? 16 : 288) : chunks <= 1536;
}
int chain_matmul(const ChainMatmul& c, cudaStream_t stream);

}  // namespace b200
