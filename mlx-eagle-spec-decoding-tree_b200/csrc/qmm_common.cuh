// Pieces shared by all quantised-matmul kernels: sizes, nibble expansion, and the rounding points of the fused epilogues.
#pragma once

#include "common.cuh"

namespace b200 {

constexpr int kChunkK = 128;          // k values one warp iteration covers
constexpr int kCounterBytes = 4096;   // head of the workspace: one int per row tile
constexpr int kMaxCounters = kCounterBytes / 4;

// The low half twice, by integer instructions: 100 x 14336 x 4096 as quantised 25.1 us, as below 25.8; 32 x 2048 x 8192 re-laid-out 6.65 and 6.8.
__device__ __forceinline__ __half2 dup_half_of_word(uint32_t u) { return u32_as_h2((u & 0xffffu) | (u << 16)); }
// (As a register pair, which the multiplications can take without a copy being made: shifted and combined it was 8 instructions a chunk; 16 x 14336 x
// 4096 as quantised 15.1 us, so 15.5.)
__device__ __forceinline__ __half2 dup_half(unsigned short bits) {
    uint32_t u;
    asm("mov.b32 %0, {%1, %1};" : "=r"(u) : "h"(bits));
    return u32_as_h2(u);
}

// 8 nibbles of one pack -> 4 half2 {e0,e4} {e1,e5} {e2,e6} {e3,e7}, each q*s+b rounded once.
__device__ __forceinline__ void dequant_pack(uint32_t w, __half2 s2, __half2 b2, uint32_t (&d)[4]) {
    constexpr uint32_t kMagic = 0x64006400u;  // fp16 1024.0 in both halves
    const __half2 k1024 = u32_as_h2(0x64006400u);
    const __half2 kSixteenth = u32_as_h2(0x2c002c00u);  // 1/16
    const __half2 kNeg64 = u32_as_h2(0xd400d400u);      // -64
    uint32_t w8 = w >> 8;
    __half2 q04 = __hsub2(u32_as_h2((w & 0x000f000fu) | kMagic), k1024);
    __half2 q15 = __hfma2(u32_as_h2((w & 0x00f000f0u) | kMagic), kSixteenth, kNeg64);
    __half2 q26 = __hsub2(u32_as_h2((w8 & 0x000f000fu) | kMagic), k1024);
    __half2 q37 = __hfma2(u32_as_h2((w8 & 0x00f000f0u) | kMagic), kSixteenth, kNeg64);
    d[0] = h2_as_u32(__hfma2(q04, s2, b2));
    d[1] = h2_as_u32(__hfma2(q15, s2, b2));
    d[2] = h2_as_u32(__hfma2(q26, s2, b2));
    d[3] = h2_as_u32(__hfma2(q37, s2, b2));
}

// Same result, bit for bit, for scales whose fp16 exponent field lies in 1..10 (2^-14 <= |s| < 2^-4; the caller
// checks this once per matrix when the weights are re-laid-out).  A nibble moved to bits 4..7 of a half IS the
// fp16 subnormal q * 2^-20, so q * s + b is one HFMA2 with s20 = s * 2^20 (exact: the product of the two is q * s,
// rounded once together with b), and s20 is the bits of s plus 20 in the exponent field.  5 integer and 6 half2
// instructions per pack instead of 5 + 8; both kinds occupy their scheduler for two cycles.
__device__ __forceinline__ void dequant_pack_fast(uint32_t w, __half2 s20, __half2 b2, uint32_t (&d)[4]) {
    constexpr uint32_t kNib = 0x00f000f0u, kLow = 0x000f000fu;
    const __half2 k16 = u32_as_h2(0x4c004c00u);
    // Two nibbles move up by an exact multiplication with 16 instead of a shift each: seven integer and four half2 instructions
    // kept the integer pipe busier (56% of its cycles) than the fp16 one (23%).
    const uint32_t w8 = w >> 8;
    d[0] = h2_as_u32(__hfma2(__hmul2(u32_as_h2(w & kLow), k16), s20, b2));
    d[1] = h2_as_u32(__hfma2(u32_as_h2(w & kNib), s20, b2));
    d[2] = h2_as_u32(__hfma2(__hmul2(u32_as_h2(w8 & kLow), k16), s20, b2));
    d[3] = h2_as_u32(__hfma2(u32_as_h2(w8 & kNib), s20, b2));
}
__device__ __forceinline__ bool fast_scale(uint32_t bits) { return ((bits >> 10) & 31u) - 1u < 10u; }   // (of the low half)
__device__ __forceinline__ __half2 scale_times_2_20(__half2 s2) { return u32_as_h2(h2_as_u32(s2) + 0x50005000u); }

__device__ __forceinline__ uint32_t comp(const uint4& v, int j) {
    return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w));
}

__device__ __forceinline__ float silu_mul_f16(float gate, float up) {
    // Rounding points of the unfused reference graph (mlx_llama.py:215): every op result is fp16.
    __half g = __float2half_rn(gate);
    __half u = __float2half_rn(up);
    float gf = __half2float(g);
    __half sig = __float2half_rn(1.0f / (1.0f + expf(-gf)));
    __half t = __hmul(g, sig);
    return __half2float(__hmul(t, u));
}


}  // namespace b200
