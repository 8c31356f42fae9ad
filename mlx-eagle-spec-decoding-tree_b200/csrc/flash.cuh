// Attention on the fifth-generation tensor cores (csrc/flash.cu) as the decode chain and prompt passes call it.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace b200 {

struct FlashArgs {
    const void* q;                 // q|k|v rows [tokens][(Hq + 2 Hkv) * HD], q rotated; query heads first
    const void* kv;                // cache as rows of HD halves
    uint64_t kv_rows;              // rows of the whole cache
    void* out;                     // [tokens][Hq * HD]
    int tokens;                    // of all requests
    int Hq, Hkv, hd, cap;          // cap: cache rows of a kv head
    float scale_log2;
    int* err;
    int polls;
    // the decode chain: `mr` tokens of each of `nreq` requests over prefix[request] committed rows, tail rows by bit mask.  Both are read before
    // the kernel ahead of the attention has ended, so nothing in the pass may write them: NULL for a causal pass of one request behind `off` rows.
    const unsigned long long* mask;
    const int* prefix;
    int nreq, mr, tail, write_off, nkb, split;
    int req_rows;                  // cache rows of one request
    // a prompt pass: causal behind `off` rows; `splits` key ranges with partial states in part_o, part_ml
    int off, splits;
    float* part_o;                 // [split][Hkv][tokens * G rows][hd]
    float* part_ml;                // [split][Hkv][rows][2]
};

// Tensor maps and launch shape of a pass; the layer comes with the launch.
struct FlashPlan {
    CUtensorMap qmap, kvmap;
    int G, heads, T, hsets, tsets, cs;           // group size; heads and tokens of a box, sets of either per kv head; cluster size
};
int flash_decode_plan(const FlashArgs& a, FlashPlan* p);
int flash_prefill_plan(const FlashArgs& a, FlashPlan* p);
// row0: first cache row of the layer's K (its V follows Hkv * cap rows on)
int flash_decode(const FlashArgs& a, const FlashPlan& p, int row0, cudaStream_t stream);
int flash_prefill(const FlashArgs& a, const FlashPlan& p, int row0, cudaStream_t stream);

}  // namespace b200
