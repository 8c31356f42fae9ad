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

constexpr int kCsPitch = 64;     // (cos, sin) of a token

// The layers of a prompt pass (embedding to the last layer's h) through the chain's kernels, tiles of 32 tokens side by side.
struct ChainPrompt {
    const b200_prefill_desc* d;  // checked
    int* err;
    const float2* cs;            // [tokens][kCsPitch], written by the first norm
    int (*norm)(const void* context, const void* weights, bool first, cudaStream_t stream);      // h -> xn; first: tokens -> h, too
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
// Whether this kernel is taken and not the large-M one: rule and figures at its definition in csrc/decode.cu.
bool chain_matmul_wins(int M, int N, int K, bool as_quantised);
int chain_matmul(const ChainMatmul& c, cudaStream_t stream);

}  // namespace b200
