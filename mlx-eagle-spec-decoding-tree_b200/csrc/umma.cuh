// Pieces shared by the kernels on the fifth-generation tensor cores (matmuls: csrc/decode.cu, csrc/qmm_gemm.cu, csrc/qmm_pair.cu; attention:
// csrc/flash.cu): matrix descriptor, completion of MMAs, and the expansion of a weight row's packs into a tensor-memory tile.
#pragma once

#include <type_traits>

#include "qmm_common.cuh"

namespace b200 {

constexpr int kRecBytes = 1152;                  // 16 rows x 128 k of the streaming layout: packs, then (scale, bias) pairs
constexpr int kRunBytes = 4 * kRecBytes;         // the four records of a 64-row block for one chunk
constexpr int kTileRows = 128;                   // weight rows of one MMA
constexpr int kTileW = 2 * kRunBytes;            // weight bytes of a row tile and chunk (both layouts: 8192 + 1024)
constexpr int kTileCols = kChunkK / 2;           // tensor-memory columns of an expanded tile: two k values per column

// K-major shared-memory matrix, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&d)[4][4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(addr),
                 "r"(d[0][0]), "r"(d[0][1]), "r"(d[0][2]), "r"(d[0][3]), "r"(d[1][0]), "r"(d[1][1]), "r"(d[1][2]), "r"(d[1][3]),
                 "r"(d[2][0]), "r"(d[2][1]), "r"(d[2][2]), "r"(d[2][3]), "r"(d[3][0]), "r"(d[3][1]), "r"(d[3][2]), "r"(d[3][3]) : "memory");
}

template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[C], uint32_t addr) {
    static_assert(C % 8 == 0 || C == 4, "columns");
    if constexpr (C % 8 == 0) {
#pragma unroll
        for (int i = 0; i < C; i += 8)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                         : "=r"(r[i]), "=r"(r[i + 1]), "=r"(r[i + 2]), "=r"(r[i + 3]), "=r"(r[i + 4]), "=r"(r[i + 5]),
                           "=r"(r[i + 6]), "=r"(r[i + 7]) : "r"(addr + i) : "memory");
    } else {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
    }
}

// The thread's row of a chunk (16 packs, 128 k) -> its lane of the tile at `trow`, sixteen columns (32 k) at a time.  Streaming layout:
// pack j of unit t is k group 4 j + t; ROWS (as quantised): pack t of unit j, its values still to be put side by side.  sc, bi: scale and
// bias of the chunk's two groups of 64, in the low halves; WORDS: doubled as words.
template <bool ROWS, bool WORDS = false>
__device__ __forceinline__ void expand_row(const uint4 (&u)[4], const uint32_t (&sc)[2], const uint32_t (&bi)[2], bool fast, uint32_t trow) {
    auto expand = [&](auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            __half2 s2 = WORDS ? dup_half_of_word(sc[j >> 1]) : dup_half((unsigned short)sc[j >> 1]);
            const __half2 b2 = WORDS ? dup_half_of_word(bi[j >> 1]) : dup_half((unsigned short)bi[j >> 1]);
            if (FAST) s2 = scale_times_2_20(s2);
            uint32_t d[4][4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t pack = ROWS ? comp(u[j], t) : comp(u[t], j);
                if (FAST) dequant_pack_fast(pack, s2, b2, d[t]);
                else dequant_pack(pack, s2, b2, d[t]);
                if (ROWS) {                              // {e0,e4} {e1,e5} {e2,e6} {e3,e7} -> adjacent k pairs
                    const uint32_t e01 = __byte_perm(d[t][0], d[t][1], 0x5410), e45 = __byte_perm(d[t][0], d[t][1], 0x7632);
                    const uint32_t e23 = __byte_perm(d[t][2], d[t][3], 0x5410), e67 = __byte_perm(d[t][2], d[t][3], 0x7632);
                    d[t][0] = e01; d[t][1] = e23; d[t][2] = e45; d[t][3] = e67;
                }
            }
            tmem_st16(trow + 16 * j, d);
        }
    };
    if (fast) expand(std::true_type{});
    else expand(std::false_type{});
}

}  // namespace b200
