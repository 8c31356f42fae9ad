// 4-bit affine quantised matmul for many token rows (prompt ingestion, the operator beyond 32 rows) on the
// fifth-generation tensor cores (tcgen05, TMEM).
//
//   y[M][N] = x[M][K] . dequant(W)[N][K]^T     (+ bias | + residual | silu(gate) * up), fp16 in, fp32 accumulate
//
// Item = (S x 128 weight rows, NT tokens, K range).  S = 2 puts two row tiles (or the gate and the up tile of the same
// rows) behind one activation tile, so an activation byte brought into shared memory feeds 256 weight rows.
//
//   2 producer warps per 128-k chunk: the weights (records of the streaming layout, or TMA boxes of the row-major layout,
//                    whose scales and biases the dequant threads load themselves, ahead) and the activations (two TMA boxes of
//                    64 k x NT rows, 128-byte swizzle, straight from row-major x; rows past M read as zero);
//   16 dequant warps in four groups that take the tiles (row tile, chunk) in turn, thread = weight row: exact q*s+b rounded
//                    once to fp16, written with tcgen05.st into the group's own tensor-memory tile (lane = weight row,
//                    column = two k values); the A operand never touches shared memory as fp16.  A group's chain (packs
//                    landed, tile free, loads, expansion, stores complete, arrival) is ~1500 cycles; four of them in
//                    flight hide it (all sixteen warps on one tile ran at 2100 cycles per chunk of two tiles);
//   MMA warp         one thread issues 8 x S tcgen05.mma (128 x NT x 16) per chunk, A from tensor memory, B from shared;
//   epilogue         the dequant warps read the accumulators (tcgen05.ld) after they have expanded the first chunks of
//                    their next item, so the tensor cores find work the moment the accumulator is free.
//
// What bounds it (S 2, NT 128, one chunk): the 16 MMAs take 1024 cycles at the tensor cores' rate; shared memory moves
// 51 KB in, 64 KB to the MMAs and 18 KB to the dequant warps, 1060 cycles at 128 bytes a cycle; the expansion issues
// ~700 of 1024 slots per scheduler.  With few tokens the weight stream is the bound: 18.4 KB per chunk are ~800 cycles of
// an SM's share of HBM.
//
// Beyond 128 tokens csrc/qmm_pair.cu, whose CTAs work in pairs on a tile, runs where it is cheaper (pair_plan below).
//
// Where the tiles alone would leave SMs idle the K range is cut across CTAs; the last CTA of a tile adds the fp32 partial
// products in split order (deterministic).  Every wait is bounded; one that runs out sets the error word.  No copy uses cluster multicast.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "b200_eagle.h"
#include "common.cuh"
#include "pipeline.cuh"
#include "qmm_common.cuh"
#include "qmm_gemm.cuh"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace b200 {
namespace {

constexpr int kDeqWarps = 16;
constexpr int kGroups = 4;                       // groups of four dequant warps, each with a tensor-memory tile of its own
constexpr int kGThreads = (kDeqWarps + 4) * 32;  // + two producer warps + two MMA warps
constexpr size_t kUmmaPartialBytes = 16u << 20;  // room for the partial products of a K split behind b200_qmm_umma
constexpr int kGemmTiles = 896;                  // tiles that a K split can hand tickets to

// Layouts of the weights
enum { W_TILED = 0, W_ROWS = 1 };

template <int S, int NT, int LAYOUT>
struct GGeo {
    static constexpr int XBYTES = NT * kChunkK * 2;                   // two boxes of 64 k
    static constexpr int STAGE = S * kTileW + XBYTES;                 // a multiple of 1024: the boxes stay swizzle-aligned
    // Row-major scales are read through L1, a 32-byte sector of a row serving eight chunks if it survives until then: half of
    // the SM's memory is left to it (64 x 4096 x 14336: 35 us with a full ring, 26 us so).
    static constexpr int FIT = LAYOUT == W_ROWS ? std::max(4, 112 * 1024 / STAGE) : (232448 - 2048) / STAGE;
    // Ring stages: an even number, so that a stage belongs to one of the two producers (and, with S = 1, to one of the two MMA
    // warps).  Even and odd chunks may drift apart; with an odd ring a wait could then meet a phase two uses away.
    static constexpr int NP = FIT < 8 ? (FIT & ~1) : 8;
    static constexpr int ACC = 2 * NT;                                // tensor-memory columns of an accumulator set: one per MMA warp
    static constexpr int NACC = ACC <= 128 ? 2 : 1;
    static constexpr int ACC0 = kGroups * kTileCols;                  // first accumulator column
    static constexpr int SMEM = NP * STAGE + 1024;                    // + alignment slack
    static_assert(STAGE % 1024 == 0 && ACC0 + NACC * ACC <= 512 && NP >= 4, "tile does not fit");
};

struct GParams {
    CUtensorMap xmap;            // x [M][K], boxes of 64 k x NT rows, 128-byte swizzle
    CUtensorMap wmap[2];         // row-major weights [N][K/8] words, boxes of 16 words x 128 rows, 64-byte swizzle (gate / up)
    const unsigned char* w[2];   // streaming layout (gate / up)
    const __half* sc[2];         // row-major layout: scales, biases [N][K/64]
    const __half* bi[2];
    int sb_pairs;                // their addresses are multiples of four: the two of a chunk can be loaded together
    const __half* bias;
    const __half* extra;         // residual [M][N] (may be y)
    __half* y;                   // [M][N]; float with B200_EPI_F32
    int* counter;                // split tickets, one per tile, zero between launches
    int* err;                    // error word or NULL
    int polls;                   // of a wait before it sets that (kNoReport without one)
    float* partial;
    int M, N, K;
    int row_items, tok_items, splits, chunks_per_split;
    int epilogue;
};

struct GItem {
    int row_item, tok0, split, c_begin, nc;
};
__device__ __forceinline__ GItem g_item(const GParams& p, int item, int NT) {
    GItem g;
    const int tok = item % p.tok_items;              // neighbouring CTAs share the weights of a row tile
    const int rest = item / p.tok_items;
    g.row_item = rest % p.row_items;
    g.split = rest / p.row_items;
    g.tok0 = tok * NT;
    g.c_begin = g.split * p.chunks_per_split;
    g.nc = min(p.chunks_per_split, p.K / kChunkK - g.c_begin);
    return g;
}

// The epilogue of one item, by the dequant warps: warp w reads lanes 32 (w % 4) .. of column group w / 4.
template <int S, int NT, bool DUAL>
__device__ __forceinline__ void gemm_epilogue(const GParams& p, const GItem& g, uint32_t acc, uint32_t accempty, int warp,
                                              int lane, int* s_last) {
    constexpr int CG = (DUAL ? NT : S * NT) / 4;         // columns (of each matrix) per warp
    constexpr int CM = (DUAL || S == 1) ? 8 : 16;        // (two accumulators per column there)
    constexpr int CH = CG < CM ? CG : CM;                // columns per trip
    const int q = warp & 3, cg = warp >> 2;
    const int s = DUAL ? 0 : (cg * CG) / NT;
    const int col0 = DUAL ? cg * CG : (cg * CG) % NT;    // first token column of the warp inside its row tile
    const int row = (DUAL ? g.row_item : g.row_item * S + s) * kTileRows + q * 32 + lane;
    const uint32_t lane_base = acc + ((uint32_t)(q * 32) << 16);
    const bool split = p.splits > 1;
    const bool both = S == 1 && g.nc > 1;                // even and odd chunks were summed apart
    const int ncol = min(CG, p.M - g.tok0 - col0);       // of them tokens
    constexpr int PR = S * kTileRows;                    // rows of a partial tile
    const size_t pstride = (size_t)p.row_items * p.tok_items * NT * PR;          // floats per split
    float* const ptile = p.partial + ((size_t)g.row_item * p.tok_items + g.tok0 / NT) * NT * PR;
    const int prow = (DUAL ? 0 : s * kTileRows) + q * 32 + lane;

    if (split) {
        // ---- partial products out: for every token column 32 consecutive floats per warp
        float* mine = ptile + (size_t)g.split * pstride + prow;
#pragma unroll 1
        for (int c0 = 0; c0 < ncol; c0 += CH) {
            uint32_t a[CH], b[CH];
            tmem_ld<CH>(a, lane_base + (DUAL ? 0 : s * NT) + col0 + c0);
            if (DUAL || both) tmem_ld<CH>(b, lane_base + NT + col0 + c0);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (both) {
#pragma unroll
                for (int i = 0; i < CH; i++) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
            }
#pragma unroll
            for (int i = 0; i < CH; i++) {
                __stcg(mine + (size_t)(col0 + c0 + i) * PR, __uint_as_float(a[i]));
                if (DUAL) __stcg(mine + (size_t)(col0 + c0 + i) * PR + kTileRows, __uint_as_float(b[i]));
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty);
        __threadfence();
        consumer_sync(kDeqWarps * 32);
        if (threadIdx.x == 0) {
            int* ctr = p.counter + g.row_item * p.tok_items + g.tok0 / NT;
            const int old = atomicAdd(ctr, 1);
            *s_last = old == p.splits - 1;
            if (old == p.splits - 1) *ctr = 0;
            __threadfence();
        }
        consumer_sync(kDeqWarps * 32);
        const bool last = *s_last;
        consumer_sync(kDeqWarps * 32);                  // read by all before the next item rewrites it
        if (!last) return;
    }
    const bool row_ok = row < p.N;
    const __half bv = (p.bias != nullptr && row_ok) ? p.bias[row] : __ushort_as_half(0);
    const bool resid = p.epilogue == B200_EPI_RESIDUAL;
    auto release = [&]() {                               // accumulator read: the MMA warp may start the next item
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty);
    };
    if (!split && ncol <= 0) release();
#pragma unroll 1
    for (int c0 = 0; c0 < ncol; c0 += CH) {
        __syncwarp();                                    // (rows past N leave the trip early)
        uint32_t a[CH], b[CH];
        if (split) {
            const float* src = ptile + prow + (size_t)(col0 + c0) * PR;
#pragma unroll
            for (int i = 0; i < CH; i++) {
                a[i] = __float_as_uint(__ldcg(src + (size_t)i * PR));
                if (DUAL) b[i] = __float_as_uint(__ldcg(src + (size_t)i * PR + kTileRows));
            }
            for (int sp = 1; sp < p.splits; sp++) {     // in split order, all loads of a trip in flight together
                const float* ss = src + (size_t)sp * pstride;
                float v[CH], w[DUAL ? CH : 1];
#pragma unroll
                for (int i = 0; i < CH; i++) {
                    v[i] = __ldcg(ss + (size_t)i * PR);
                    if (DUAL) w[i] = __ldcg(ss + (size_t)i * PR + kTileRows);
                }
#pragma unroll
                for (int i = 0; i < CH; i++) {
                    a[i] = __float_as_uint(__uint_as_float(a[i]) + v[i]);
                    if (DUAL) b[i] = __float_as_uint(__uint_as_float(b[i]) + w[i]);
                }
            }
        } else {
            tmem_ld<CH>(a, lane_base + (DUAL ? 0 : s * NT) + col0 + c0);
            if (DUAL || both) tmem_ld<CH>(b, lane_base + NT + col0 + c0);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (both) {
#pragma unroll
                for (int i = 0; i < CH; i++) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
            }
            if (c0 + CH >= ncol) release();
        }
        const int tok = g.tok0 + col0 + c0;
        if (!row_ok) continue;
        __half* dst = p.y + (size_t)tok * p.N + row;
        const int cnt = min(CH, p.M - tok);
        if (resid) {
            const __half* rs = p.extra + (size_t)tok * p.N + row;
            unsigned short r[CH];
#pragma unroll
            for (int i = 0; i < CH; i++) r[i] = i < cnt ? __ldcg(reinterpret_cast<const unsigned short*>(rs) + (size_t)i * p.N) : 0;
#pragma unroll
            for (int i = 0; i < CH; i++)
                if (i < cnt) {
                    __half o = __float2half_rn(__uint_as_float(a[i]));
                    if (p.bias != nullptr) o = __hadd(o, bv);
                    dst[(size_t)i * p.N] = __hadd(__ushort_as_half(r[i]), o);
                }
        } else if (DUAL) {
#pragma unroll
            for (int i = 0; i < CH; i++)
                if (i < cnt) dst[(size_t)i * p.N] = __float2half_rn(silu_mul_f16(__uint_as_float(a[i]), __uint_as_float(b[i])));
        } else if (p.epilogue == B200_EPI_F32) {
            float* out = reinterpret_cast<float*>(p.y) + (size_t)tok * p.N + row;
#pragma unroll
            for (int i = 0; i < CH; i++)
                if (i < cnt) out[(size_t)i * p.N] = __uint_as_float(a[i]);
        } else {
#pragma unroll
            for (int i = 0; i < CH; i++)
                if (i < cnt) {
                    __half o = __float2half_rn(__uint_as_float(a[i]));
                    if (p.bias != nullptr) o = __hadd(o, bv);
                    dst[(size_t)i * p.N] = o;
                }
        }
    }
}

template <int S, int NT, bool DUAL, int LAYOUT>
__global__ void __launch_bounds__(kGThreads, 1) qmm_gemm_kernel(const __grid_constant__ GParams p) {
    using G = GGeo<S, NT, LAYOUT>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    __shared__ uint64_t s_bars[2 * 8 + 2 * kGroups + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;
    uint64_t* pfull = s_bars;                        // stage landed            (producer -> dequant warps, MMA warp)
    uint64_t* pempty = pfull + G::NP;                // stage read              (S groups of warps + the MMAs -> producer)
    uint64_t* tready = pempty + G::NP;               // tile expanded           (a group's 4 warps -> MMA warp)
    uint64_t* tfree = tready + kGroups;              // tile's MMAs complete    (tcgen05.commit -> the group)
    uint64_t* accfull = tfree + kGroups;             // accumulators complete   (tcgen05.commit -> epilogue)
    uint64_t* accempty = accfull + G::NACC;          // accumulators read       (16 warps -> MMA warp)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nitems = p.row_items * p.tok_items * p.splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::NP; s++) {
            mbar_init(smem_u32(pfull + s), 1);
            mbar_init(smem_u32(pempty + s), 4 * S + S);
        }
        for (int s = 0; s < kGroups; s++) {
            mbar_init(smem_u32(tready + s), 4);
            mbar_init(smem_u32(tfree + s), 1);
        }
        for (int s = 0; s < G::NACC; s++) {
            mbar_init(smem_u32(accfull + s), 2);
            mbar_init(smem_u32(accempty + s), kDeqWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == kDeqWarps + 2) {                     // the first MMA warp owns the tensor memory (all 512 columns)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    auto gwait = [&](const uint64_t* bar, uint32_t parity, int code) {
        mbar_wait_reported(smem_u32(bar), parity, p.polls, p.err, code);
        __syncwarp();
    };
    pdl_launch_dependents();

    if (warp >= kDeqWarps && warp < kDeqWarps + 2) {
        // ------------------------------------------------------------------ producers: warp i asks for the chunks with number % 2 == i
        const uint32_t par = __shfl_sync(0xffffffffu, warp - kDeqWarps, 0);
        const int nchunks = p.K / kChunkK;
        const int nblocks = (p.N + 63) / 64;
        bool waited = LAYOUT == W_ROWS;              // (row-major weights may come from the kernel before this one)
        if (waited) pdl_wait();
        uint32_t n = 0;                              // chunks of earlier items
        uint32_t pend = 0;                           // stages of this warp whose activations are still to be asked for
        auto load_x = [&](uint32_t s, int c, int tok0) {
            const uint32_t dst = smem_u32(ring + s * G::STAGE + S * kTileW), bar = smem_u32(pfull + s);
            tma_box(dst, &p.xmap, c * kChunkK, tok0, bar);
            tma_box(dst + NT * 128, &p.xmap, c * kChunkK + 64, tok0, bar);
        };
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            const GItem g = g_item(p, item, NT);
            int c = (int)((par - n) & 1u);
            // the item's 64-row blocks, one run of 4608 bytes each per chunk (gate blocks, then up blocks)
            const unsigned char* wsrc[2 * S];
#pragma unroll
            for (int i = 0; i < 2 * S; i++)
                wsrc[i] = p.w[DUAL ? i >> 1 : 0] +
                          ((size_t)min(DUAL ? g.row_item * 2 + (i & 1) : g.row_item * 2 * S + i, nblocks - 1) * nchunks + g.c_begin + c) * kRunBytes;
            for (; c < g.nc; c += 2) {
                const uint32_t slot = (n + c) % G::NP, use = (n + c) / G::NP;
                if (use > 0) gwait(pempty + slot, (use - 1) & 1u, 1);
                const uint32_t bar = smem_u32(pfull + slot);
                unsigned char* stage = ring + slot * G::STAGE;
                if (elect_one()) {
                    mbar_expect_tx(bar, LAYOUT == W_TILED ? G::STAGE : S * 8192 + G::XBYTES);
                    if (LAYOUT == W_TILED) {
#pragma unroll
                        for (int i = 0; i < 2 * S; i++) bulk_copy_g2s(smem_u32(stage + i * kRunBytes), wsrc[i], kRunBytes, bar);
                    } else {
#pragma unroll
                        for (int i = 0; i < S; i++)
                            tma_box(smem_u32(stage + i * kTileW), &p.wmap[DUAL ? i : 0], (g.c_begin + c) * 16,
                                    (DUAL ? g.row_item : g.row_item * S + i) * kTileRows, bar);
                    }
                    if (waited) load_x(slot, g.c_begin + c, g.tok0);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 2 * S; i++) wsrc[i] += 2 * kRunBytes;
                if (!waited) {
                    // the first stages' weights do not depend on the kernel before this one, the activations do
                    pend++;
                    if (c + 2 >= min(g.nc, (int)G::NP)) {
                        pdl_wait();
                        waited = true;
                        if (elect_one())
                            for (uint32_t i = 0; i < pend; i++) load_x(par + 2 * i, g.c_begin + (int)(par + 2 * i), g.tok0);
                        __syncwarp();
                    }
                }
            }
            n += g.nc;
            if (!waited) { pdl_wait(); waited = true; }       // (a first item of one chunk leaves the second warp without)
        }
        if (!waited) pdl_wait();
    } else if (warp >= kDeqWarps + 2) {
        // ------------------------------------------------------------------ MMA issuers (an elected thread each): S = 2: one per row
        // tile, S = 1: even and odd chunks, each into an accumulator of its own; while one stands at a barrier after its eight
        // MMAs (~190 cycles) the other's run.
        const uint32_t me = __shfl_sync(0xffffffffu, warp - (kDeqWarps + 2), 0);
        const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
        uint32_t n = 0, it = 0;                          // chunks of earlier items, items
        for (int item = blockIdx.x; item < nitems; item += gridDim.x, it++) {
            const GItem g = g_item(p, item, NT);
            const uint32_t ab = it % G::NACC, ause = it / G::NACC;
            if (ause > 0) gwait(accempty + ab, (ause - 1) & 1u, 2);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t d0 = tmem + G::ACC0 + ab * G::ACC + me * NT;
            bool first = true;
            for (int c = S == 2 ? 0 : (int)me; c < g.nc; c += S == 2 ? 1 : 2) {
                const uint32_t tile = (n + c) * S + (S == 2 ? me : 0);            // tile number: group and use of its tensor-memory tile
                const uint32_t ts = tile % kGroups, slot = (n + c) % G::NP;
                // (the expanded tile is ready only after its group has seen the whole stage land, the activations included)
                gwait(tready + ts, (tile / kGroups) & 1u, 2);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t b0 = sw128_desc(smem_u32(ring + slot * G::STAGE + S * kTileW));
                const uint32_t a0 = tmem + ts * kTileCols;
                if (elect_one()) {
                    const uint32_t accumulate = first ? 0u : 1u;
#pragma unroll
                    for (int ks = 0; ks < kChunkK / 16; ks++)
                        asm volatile(
                            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d0),
                            "r"(a0 + ks * 8), "l"(b0 + ((ks >> 2) * (NT * 128) + (ks & 3) * 32) / 16), "r"(idesc), "r"(ks == 0 ? accumulate : 1u)
                            : "memory");
                    commit_to(smem_u32(tfree + ts));
                    commit_to(smem_u32(pempty + slot));
                }
                __syncwarp();
                first = false;
            }
            if (elect_one()) commit_to(smem_u32(accfull + ab));
            __syncwarp();
            n += g.nc;
        }
    } else {
        // ------------------------------------------------------------------ dequant warps + epilogue
        const int q = warp & 3;
        const uint32_t grp = warp >> 2;                   // takes the tiles with number % 4 == grp, into tensor-memory tile grp
        const int r = q * 32 + lane;                      // weight row inside the tile = tensor-memory lane
        const int rr = r & 15;
        const uint32_t rowoff = LAYOUT == W_TILED ? ((r >> 6) * kRunBytes + ((r >> 4) & 3) * kRecBytes + (rr >> 3) * 512 + (rr & 7) * 64) : r * 64;
        const uint32_t scoff = (r >> 6) * kRunBytes + ((r >> 4) & 3) * kRecBytes + 1024 + rr * 8;
        const uint32_t trow = tmem + grp * kTileCols + ((uint32_t)(q * 32) << 16);
        // Row-major layout: this row's scales and biases of a chunk, loaded one tile ahead.
        uint32_t sb_s = 0, sb_b = 0;
        auto load_sb = [&](const GItem& g, uint32_t k) {
            const uint32_t s = k % S;
            const int tile_row = DUAL ? g.row_item : g.row_item * S + (int)s;
            const size_t e = (size_t)min(tile_row * kTileRows + r, p.N - 1) * (p.K / 64) + (g.c_begin + k / S) * 2;
            const __half *sp = p.sc[DUAL ? s : 0] + e, *bp = p.bi[DUAL ? s : 0] + e;
            if (p.sb_pairs) {
                sb_s = __ldg(reinterpret_cast<const uint32_t*>(sp));
                sb_b = __ldg(reinterpret_cast<const uint32_t*>(bp));
            } else {
                const unsigned short *su = reinterpret_cast<const unsigned short*>(sp), *bu = reinterpret_cast<const unsigned short*>(bp);
                sb_s = __ldg(su) | (uint32_t)__ldg(su + 1) << 16;
                sb_b = __ldg(bu) | (uint32_t)__ldg(bu + 1) << 16;
            }
        };
        if (LAYOUT == W_ROWS) pdl_wait();                 // (the kernel before this one may have written the weights)
        uint32_t cbase = 0, tbase = 0, tuse = 0, it = 0;  // chunks and tiles of earlier items, tiles of this group so far, items
        bool pending = false;
        GItem prev{};
        auto epilogue = [&]() {
            const uint32_t ab = (it - 1) % G::NACC;
            gwait(accfull + ab, ((it - 1) / G::NACC) & 1u, 3);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            gemm_epilogue<S, NT, DUAL>(p, prev, tmem + G::ACC0 + ab * G::ACC, smem_u32(accempty + ab), warp, lane, &s_last);
            pending = false;
        };
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            const GItem g = g_item(p, item, NT);
            const uint32_t ntiles = g.nc * S;
            const uint32_t k0 = (grp - tbase) & (kGroups - 1);
            if (LAYOUT == W_ROWS && k0 < ntiles) load_sb(g, k0);
            for (uint32_t k = k0; k < ntiles; k += kGroups, tuse++) {
                const uint32_t n = cbase + k / S, s = k % S;
                const uint32_t slot = n % G::NP;
                gwait(pfull + slot, (n / G::NP) & 1u, 3);
                if (tuse > 0) gwait(tfree + grp, (tuse - 1) & 1u, 3);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const unsigned char* tile = ring + slot * G::STAGE + s * kTileW;
                uint4 u[4];
                uint32_t sc2[2], bi2[2];              // scale, bias of the chunk's two k groups, low halves
                if (LAYOUT == W_TILED) {
                    // rows are 64 bytes apart: every other pair of rows reads its 16-byte units in the other order, so that
                    // eight lanes meet in the same banks in pairs only
                    const int flip = (r >> 1) & 1;
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {
                        const uint4 a = *reinterpret_cast<const uint4*>(tile + rowoff + (i + flip) * 16);
                        const uint4 b = *reinterpret_cast<const uint4*>(tile + rowoff + (i + 1 - flip) * 16);
                        u[i] = flip ? b : a;
                        u[i + 1] = flip ? a : b;
                    }
                    const uint2 sb = *reinterpret_cast<const uint2*>(tile + scoff);
                    sc2[0] = sb.x; bi2[0] = sb.x >> 16;
                    sc2[1] = sb.y; bi2[1] = sb.y >> 16;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        u[i] = *reinterpret_cast<const uint4*>(tile + rowoff + ((i ^ ((r >> 1) & 3)) << 4));
                    const uint32_t sv = sb_s, bv = sb_b;
                    if (k + kGroups < ntiles) load_sb(g, k + kGroups);
                    sc2[0] = sv; sc2[1] = sv >> 16;
                    bi2[0] = bv; bi2[1] = bv >> 16;
                }
                const bool fast = __all_sync(0xffffffffu, fast_scale(sc2[0]) && fast_scale(sc2[1]));
                expand_row<LAYOUT == W_ROWS, LAYOUT == W_ROWS && NT == 128>(u, sc2, bi2, fast, trow);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(pempty + slot));       // the packs are in registers
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(tready + grp));
                // the item before this one: its epilogue runs once this warp's first tile of this item is expanded
                if (pending) epilogue();
            }
            if (pending) epilogue();
            cbase += g.nc;
            tbase += ntiles;
            prev = g;
            pending = true;
            it++;
            if (it == 1) pdl_wait();                      // before this thread's first global access
        }
        if (pending) epilogue();
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == kDeqWarps + 2)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

// ---- work split: token columns per item, row tiles behind one activation tile, K ranges
struct GPlan {
    int S, NT, splits, cps, row_items, tok_items;
    double cost;
};

size_t gemm_partial_bytes(const GPlan& pl) {
    return pl.splits > 1 ? (size_t)pl.splits * pl.row_items * pl.tok_items * pl.NT * pl.S * kTileRows * sizeof(float) : 0;
}

// Cost in SM cycles, fitted to measurements on B200 (M 16 .. 1024; N x K of a few thousand): a chunk of one / two row tiles
// costs 480 / 900 + 5 per token column, an item its fill and epilogue, a K split the partial products out and in (38 bytes a
// cycle) and the ticket, a launch ~9000.
GPlan gemm_plan(int M, int N, int K, bool dual, int sms, size_t partial_room) {
    GPlan best{};
    double best_cost = 1e30;
    const int nchunks = K / kChunkK;
    for (int NT = 16; NT <= 128; NT *= 2) {
        if (NT < 128 && NT / 2 >= M && NT > 16) break;               // half the columns would do
        for (int S = dual ? 2 : 1; S <= 2; S++) {
            const int rows = dual ? kTileRows : S * kTileRows;
            GPlan pl{};
            pl.S = S; pl.NT = NT;
            pl.row_items = (N + rows - 1) / rows;
            pl.tok_items = (M + NT - 1) / NT;
            const long long tiles = (long long)pl.row_items * pl.tok_items;
            const double chunk = (S == 2 ? 900.0 : 480.0) + 5.0 * NT;
            for (int splits = 1; splits <= std::max(1, nchunks / 2); splits++) {
                if (splits > 1 && (tiles > kGemmTiles || splits > 32)) break;
                pl.cps = (nchunks + splits - 1) / splits;
                pl.splits = (nchunks + pl.cps - 1) / pl.cps;
                if (pl.splits != splits) continue;
                if (splits > 1 && gemm_partial_bytes(pl) > partial_room) break;
                const long long rounds = (tiles * splits + sms - 1) / sms;
                const double out = std::min(NT, (M + 15) & ~15) * S * 128 * 4.0 / 38.0;    // partial products of an item, cycles
                const double cost = 9000 + rounds * (pl.cps * chunk + 700 + NT * S * 4.0) + (splits > 1 ? 3400 + rounds * out + out * splits : 0.0);
                if (cost < best_cost) { best_cost = cost; best = pl; }
                if (tiles * splits >= 3LL * sms) break;
            }
        }
    }
    best.cost = best_cost;
    return best;
}

// The same for csrc/qmm_pair.cu (more than 128 rows), whose work is dealt to pairs of SMs; of the two kernels the cheaper one runs.  Fitted to
// 26 shapes of 129 to 1024 rows: a chunk costs its MMAs, 4 cycles a token, or the expansion; an item that drains behind the last
// MMAs 23 cycles a token; a K split 6600 and 12.7 cycles a token and range.  Pairs win where a weight is used by more than 128 tokens and
// the K of an item is long (203 x 4096 x 14336: 42 -> 32 us, 517 x 6144 x 4096: 28 -> 23, 1024 x 4096 x 14336: 92 -> 85); where the start and the end
// of a kernel are most of it, one CTA's shorter ones do (256 x 3584 x 3584: 13.4 against 16.4 us, 256 x 1024 x 1024: 6 against 10).
size_t pair_partial_bytes(const PairPlan& pl) {
    return pl.splits > 1 ? (size_t)pl.splits * pl.row_items * pl.tok_items * pl.NT * 2 * kTileRows * sizeof(float) : 0;
}

PairPlan pair_plan(int M, int N, int K, bool dual, int sms, size_t partial_room) {
    PairPlan best{};
    best.cost = 1e30;
    if (M <= 128) return best;
    const int nchunks = K / kChunkK, pairs = std::max(1, sms / 2), rows = dual ? kTileRows : 2 * kTileRows;
    for (int t = (M + 255) / 256; t <= (M + 127) / 128; t++) {
        PairPlan pl{};
        pl.tok_items = t;
        pl.NT = ((M + t - 1) / t + 31) / 32 * 32;
        pl.row_items = (N + rows - 1) / rows;
        const long long tiles = (long long)pl.row_items * t;
        const double chunk = std::max(4.0 * pl.NT, 800.0);
        for (int splits = 1; splits <= std::max(1, nchunks / 2); splits++) {
            if (splits > 1 && (2 * tiles > kGemmTiles || splits > 32)) break;
            pl.cps = (nchunks + splits - 1) / splits;
            pl.splits = (nchunks + pl.cps - 1) / pl.cps;
            if (pl.splits != splits) continue;
            if (splits > 1 && pair_partial_bytes(pl) > partial_room) break;
            const long long rounds = (tiles * splits + pairs - 1) / pairs;
            const double cost = 9500 + rounds * (pl.cps * chunk + 1140) + 23.0 * pl.NT + (splits > 1 ? 6600 + rounds * splits * 12.7 * pl.NT : 0.0);
            if (cost < best.cost) { best = pl; best.cost = cost; }
            if (tiles * splits >= 3LL * pairs) break;
        }
    }
    return best;
}

template <int S, int NT, bool DUAL, int LAYOUT>
int launch_gemm(const GParams& p, int sms, cudaStream_t stream) {
    auto kern = qmm_gemm_kernel<S, NT, DUAL, LAYOUT>;
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(kern, GGeo<S, NT, LAYOUT>::SMEM, done)) return check_launch();
    const int nitems = p.row_items * p.tok_items * p.splits;
    launch_kernel(kern, dim3(nitems < sms ? nitems : sms), dim3(kGThreads), (size_t)GGeo<S, NT, LAYOUT>::SMEM, stream, p);
    return check_launch();
}

template <int S, bool DUAL, int LAYOUT>
int launch_gemm_nt(const GParams& p, int nt, int sms, cudaStream_t stream) {
    switch (nt) {
        case 16: return launch_gemm<S, 16, DUAL, LAYOUT>(p, sms, stream);
        case 32: return launch_gemm<S, 32, DUAL, LAYOUT>(p, sms, stream);
        case 64: return launch_gemm<S, 64, DUAL, LAYOUT>(p, sms, stream);
        default: return launch_gemm<S, 128, DUAL, LAYOUT>(p, sms, stream);
    }
}

}  // namespace

int gemm_sms() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if ((n = known[dev & 63].load(std::memory_order_relaxed)) > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    known[dev & 63].store(n, std::memory_order_relaxed);
    return n;
}

size_t qmm_gemm_partial_bytes(int M, int N, int K, bool dual) {
    const int sms = gemm_sms();
    const size_t room = (size_t)1 << 40;
    const GPlan one = gemm_plan(M, N, K, dual, sms, room);
    const PairPlan two = pair_plan(M, N, K, dual, sms, room);
    return std::max(gemm_partial_bytes(one), two.cost < 0.95 * one.cost ? pair_partial_bytes(two) : 0);
}

int qmm_gemm(const GemmArgs& a, cudaStream_t stream) {
    const bool dual = a.epilogue == B200_EPI_SILU_MUL, tiled = a.w_tiled != nullptr;
    const int sms = gemm_sms();
    const GPlan pl = gemm_plan(a.M, a.N, a.K, dual, sms, a.partial_bytes);
    const PairPlan pairs = pair_plan(a.M, a.N, a.K, dual, sms, a.partial_bytes);
    if (pairs.cost < 0.95 * pl.cost && a.epilogue != B200_EPI_F32 && (tiled || !dual)) return qmm_pair(a, pairs, stream);
    GParams p{};
    int rc = make_map_2d(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, (uint64_t)a.K, (uint64_t)a.M, (uint64_t)a.K * 2, 64, (uint32_t)pl.NT,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200_OK) return rc;
    for (int i = 0; !tiled && i < (dual ? 2 : 1); i++) {
        rc = make_map_2d(&p.wmap[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, a.wq[i], (uint64_t)a.K / 8, (uint64_t)a.N, (uint64_t)a.K / 2, 16, kTileRows,
                         CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (rc != B200_OK) return rc;
    }
    p.w[0] = static_cast<const unsigned char*>(a.w_tiled);
    p.w[1] = static_cast<const unsigned char*>(a.w2_tiled);
    p.sb_pairs = 1;
    for (int i = 0; i < 2; i++) {
        p.sc[i] = static_cast<const __half*>(a.scales[i]);
        p.bi[i] = static_cast<const __half*>(a.biases[i]);
        if ((reinterpret_cast<uintptr_t>(a.scales[i]) | reinterpret_cast<uintptr_t>(a.biases[i])) & 3u) p.sb_pairs = 0;
    }
    p.bias = static_cast<const __half*>(a.bias);
    p.extra = static_cast<const __half*>(a.extra);
    p.y = static_cast<__half*>(a.y);
    p.counter = a.counters;
    p.err = a.err;
    p.polls = a.err != nullptr ? wait_polls(kWaitPolls, kFirmPolls / 2) : kNoReport;
    p.partial = static_cast<float*>(a.partial);
    p.M = a.M; p.N = a.N; p.K = a.K;
    p.row_items = pl.row_items; p.tok_items = pl.tok_items; p.splits = pl.splits; p.chunks_per_split = pl.cps;
    p.epilogue = a.epilogue;
    if (dual) return tiled ? launch_gemm_nt<2, true, W_TILED>(p, pl.NT, sms, stream) : launch_gemm_nt<2, true, W_ROWS>(p, pl.NT, sms, stream);
    if (tiled) return pl.S == 2 ? launch_gemm_nt<2, false, W_TILED>(p, pl.NT, sms, stream) : launch_gemm_nt<1, false, W_TILED>(p, pl.NT, sms, stream);
    return pl.S == 2 ? launch_gemm_nt<2, false, W_ROWS>(p, pl.NT, sms, stream) : launch_gemm_nt<1, false, W_ROWS>(p, pl.NT, sms, stream);
}

}  // namespace b200

extern "C" {

using namespace b200;

size_t b200_qmm_gemm_workspace_bytes(int M, int N, int K, int epilogue) {
    if (M < 1 || N < 8 || (N % 8) != 0 || K < kChunkK || (K % kChunkK) != 0) return 0;
    return kCounterBytes + qmm_gemm_partial_bytes(M, N, K, epilogue == B200_EPI_SILU_MUL);
}

int b200_qmm_gemm(const void* x, const void* wt, const void* wt2, const void* bias, const void* extra, void* y, int M, int N, int K,
                  int epilogue, void* workspace, size_t workspace_bytes, void* stream) {
    if (M < 1 || N < 8 || (N % 8) != 0 || K < kChunkK || (K % kChunkK) != 0) return B200_EINVAL;
    if (epilogue < B200_EPI_NONE || epilogue > B200_EPI_SILU_MUL) return B200_EINVAL;
    const bool dual = epilogue == B200_EPI_SILU_MUL;
    if (!x || !wt || !y || !workspace || (dual && (!wt2 || bias)) || (epilogue == B200_EPI_RESIDUAL && (!extra || bias))) return B200_EINVAL;
    if (!aligned16(x) || !aligned16(wt) || !aligned16(wt2) || !aligned16(y) || !aligned16(bias) || !aligned16(extra) || !aligned16(workspace))
        return B200_EALIGN;
    if (workspace_bytes < (size_t)kCounterBytes) return B200_EWORKSPACE;
    GemmArgs a{};
    a.x = x; a.w_tiled = wt; a.w2_tiled = wt2; a.bias = bias; a.extra = extra; a.y = y;
    a.M = M; a.N = N; a.K = K; a.epilogue = epilogue;
    gemm_workspace(a, workspace, workspace_bytes);
    return qmm_gemm(a, static_cast<cudaStream_t>(stream));
}

// The fixed form of round row counts: up to 128 rows, whole 128-row tiles, the error word first in the workspace.
size_t b200_qmm_umma_workspace_bytes(int M, int K) {
    if (M < 1 || M > 128 || K < kChunkK || (K % kChunkK) != 0) return 0;
    return kCounterBytes + kUmmaPartialBytes;
}

int b200_qmm_umma(const void* x, const void* w_tiled, const void* bias, void* y, int M, int N, int K, void* workspace,
                  size_t workspace_bytes, void* stream) {
    if (!x || !w_tiled || !y || !workspace || M < 1 || M > 128 || N < kTileRows || K < kChunkK) return B200_EINVAL;
    if ((N % kTileRows) != 0 || (K % kChunkK) != 0) return B200_EUNSUPPORTED;
    if (!aligned16(x) || !aligned16(w_tiled) || !aligned16(y) || !aligned16(workspace) || !aligned16(bias)) return B200_EALIGN;
    if (workspace_bytes < b200_qmm_umma_workspace_bytes(M, K)) return B200_EWORKSPACE;
    GemmArgs a{};
    a.x = x; a.w_tiled = w_tiled; a.bias = bias; a.y = y;
    a.M = M; a.N = N; a.K = K; a.epilogue = B200_EPI_NONE;
    gemm_workspace(a, workspace, workspace_bytes);
    a.err = static_cast<int*>(workspace);
    a.counters = static_cast<int*>(workspace) + 64;
    return qmm_gemm(a, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
