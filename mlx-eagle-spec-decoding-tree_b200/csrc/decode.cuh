// The kernel chain of a forward pass (csrc/decode.cu) as csrc/forward.cu calls it.
#pragma once

#include "common.cuh"

namespace b200 {

// What b200_forward has checked and laid out of the descriptor: everything is valid, tp_world <= 1.
struct ChainArgs {
    const b200_forward_desc* d;
    const void* const* layers;   // host copy of the layer table
    int* err;             // error word
    float* ssq;           // [hidden / 32][32]
    float2* cs;           // [32][64]
    int splits[5];        // K split (cluster size) asked for per phase A, C, D, E, head; 0 = planner
};

int forward_chain(const ChainArgs& a, cudaStream_t stream);

// y[M][N] = x[M][K] . W^T (+ bias), M <= 32, W in the streaming layout, by the chain's matmul kernel on its own.
int chain_matmul(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, int* err, cudaStream_t stream);

}  // namespace b200
