// 4-bit affine quantised matmul for more than 128 token rows, a pair of CTAs (cta_group::2) to a tile of 256 weight rows and up to
// 256 tokens.
//
//   y[M][N] = x[M][K] . dequant(W)[N][K]^T     (+ bias | + residual | silu(gate) * up), fp16 in, fp32 accumulate
//
// Why pairs: beyond 128 tokens csrc/qmm_gemm.cu expands every weight once per 128 tokens, and its two row tiles a chunk kept the
// schedulers (700 issue slots of 1024) and shared memory (1060 cycles) as busy as the tensor cores.  Here a CTA expands its 128
// rows of a chunk once for all the tile's tokens into its own tensor memory, and brings in half of the tokens' activations, which
// the MMAs of both CTAs read: half the expansion and half the shared-memory traffic per product.
//
//   producer warps   per 128-k chunk: the CTA's weights (two 64-row blocks; gate and up: one each); two boxes of 64 k x NT / 2
//                    tokens, straight from row-major x (rows past M read as zero);
//   16 dequant warps in four groups that take the chunks in turn, thread = weight row (see csrc/qmm_gemm.cu);
//   MMA warp         of the even CTA: eight tcgen05.mma (256 x NT x 16) a chunk for both, A from tensor memory, B from the two
//                    CTAs' shared memory; completion is reported to both;
//   epilogue         the dequant warps, once they have expanded their first chunk of the next item: accumulators to registers
//                    (as fp16: every epilogue rounds the product first), which frees them, then the output.
//
// NT (a multiple of 32) follows the row count: M tokens in ceil(M / 256) or more tiles of equal size.  What bounds it: the MMAs, 4 NT cycles a
// chunk, from about 128 tokens a tile on; below that the expansion, ~450.
//
// Where tiles are few the K range is cut across pairs as in csrc/qmm_gemm.cu.  Every wait is bounded; one that runs out sets the error
// word and goes on.  No copy uses cluster multicast (the MMAs' completion does).
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>

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
constexpr int kAcc0 = kGroups * kTileCols;       // first accumulator column
constexpr int kThreads = (kDeqWarps + 3) * 32;   // + weight producer, activation producer, MMA issuer
constexpr int kMaxNT = 256;
// Layouts of the weights: re-laid-out, or as quantised with scales and biases loaded by the dequant threads (W_ROWS) or as boxes of 16
// bytes a row, the four chunks around (W_BOXES: where TMA can address them, K a multiple of 512).  Through L1 the two loads a thread and
// chunk, 32 lines each, took 5 us of the 36 of 203 x 4096 x 14336.
enum { W_TILED = 0, W_ROWS = 1, W_BOXES = 2 };

template <bool DUAL, int LAYOUT>
struct PGeo {
    static constexpr int X = kMaxNT / 2 * kChunkK * 2;                 // activations of a chunk: two boxes of 64 k
    // Rings of their own: an activation stage is in use from its load to the chunk's MMAs, a weight stage only until it has been expanded,
    // and that begins long before.  (One ring of five stages for both ran at 0.75 us a chunk of 256 tokens, whatever they were.)
    // Row-major scales are read through L1, which some memory is left to (see GGeo).
    static constexpr int NX = LAYOUT == W_ROWS ? 4 : 5;
    static constexpr int NW = LAYOUT == W_ROWS ? 4 : (LAYOUT == W_BOXES || DUAL ? 5 : 6);
    static constexpr int WSTAGE = LAYOUT == W_BOXES ? 8192 + 2 * kTileRows * 16 : kTileW;
    static constexpr int W0 = NX * X;
    static constexpr int SWAP = W0 + NW * WSTAGE;                     // gate / up: what two warps hand each other, two units of 16 bytes a thread
    static constexpr int SMEM = SWAP + (DUAL ? 2 * kDeqWarps * 32 * 16 : 0) + 1024;
    static_assert(W0 % 1024 == 0 && WSTAGE % 1024 == 0 && !(DUAL && LAYOUT != W_TILED) && kAcc0 + kMaxNT <= 512 && SMEM + 1024 <= 232448, "tile does not fit");
};

struct PairParams {
    CUtensorMap xmap;            // x [M][K], boxes of 64 k x NT / 2 rows, 128-byte swizzle
    CUtensorMap wmap;            // row-major weights [N][K/8] words, boxes of 16 words x 128 rows, 64-byte swizzle
    CUtensorMap smap, bmap;      // W_BOXES: scales, biases [N][K/64], boxes of 8 x 128 rows
    const unsigned char* w[2];   // streaming layout (gate / up)
    const __half* sc;            // row-major layout: scales, biases [N][K/64]
    const __half* bi;
    int sb_pairs;                // their addresses are multiples of four: the two of a chunk can be loaded together
    const __half* bias;
    const __half* extra;         // residual [M][N] (may be y)
    __half* y;                   // [M][N]
    int* counter;                // split tickets, two per tile, zero between launches
    int* err;
    int polls;
    float* partial;              // [split][tile][CTA of the pair][four tokens][128 rows][4]
    int M, N, K, NT;
    int row_items, tok_items, splits, chunks_per_split;
    int epilogue;
};

struct PItem {
    int row_item, tok0, split, c_begin, nc, tile;
};
__device__ __forceinline__ PItem p_item(const PairParams& p, int item) {
    PItem g;
    const int tok = item % p.tok_items;              // neighbouring pairs share the weights of a row tile
    const int rest = item / p.tok_items;
    g.row_item = rest % p.row_items;
    g.split = rest / p.row_items;
    g.tok0 = tok * p.NT;
    g.tile = g.row_item * p.tok_items + tok;
    g.c_begin = g.split * p.chunks_per_split;
    g.nc = min(p.chunks_per_split, p.K / kChunkK - g.c_begin);
    return g;
}

__device__ __forceinline__ void commit_to_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// At a barrier of either CTA.  What passes between the two is tensor memory, ordered by the tcgen05 fences around this, and word of copies that
// have landed, so the arrival needs no more than its own order: one that releases to the cluster, and waits that acquire from it,
// make memory coherent between SMs and took 0.35 us of every chunk.
__device__ __forceinline__ void arrive_pair(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory"); }

template <bool DUAL, int LAYOUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) qmm_pair_kernel(const __grid_constant__ PairParams p) {
    using G = PGeo<DUAL, LAYOUT>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    __shared__ uint64_t wfull[G::NW], wempty[G::NW]; // weights landed (-> dequant warps), expanded (a group's 4 warps -> producer)
    __shared__ uint64_t xfull[G::NX], xempty[G::NX]; // activations landed (-> MMA warp), read (the MMAs -> producer)
    __shared__ uint64_t xpeer[G::NX];                // the odd CTA's activations landed (its MMA warp -> the even one's)
    __shared__ uint64_t tready[kGroups];             // tile expanded, both CTAs (2 x 4 warps -> the even CTA's MMA warp)
    __shared__ uint64_t tfree[kGroups];              // tile's MMAs complete    (-> the group)
    __shared__ uint64_t accfull, accempty;           // accumulators complete (-> epilogue) and read (2 x 16 warps -> MMA warp)
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int nitems = p.row_items * p.tok_items * p.splits, first_item = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::NW; s++) {
            mbar_init(smem_u32(wfull + s), 1);
            mbar_init(smem_u32(wempty + s), 4);
        }
        for (int s = 0; s < G::NX; s++) {
            mbar_init(smem_u32(xfull + s), 1);
            mbar_init(smem_u32(xempty + s), 1);
            mbar_init(smem_u32(xpeer + s), 1);
        }
        for (int s = 0; s < kGroups; s++) {
            mbar_init(smem_u32(tready + s), 8);
            mbar_init(smem_u32(tfree + s), 1);
        }
        mbar_init(smem_u32(&accfull), 1);
        mbar_init(smem_u32(&accempty), 2 * kDeqWarps);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == kDeqWarps + 2) {                     // the MMA warps take all tensor memory of the pair
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cluster_arrive_relaxed();                        // the barriers of both are there before either is arrived at
    cluster_wait();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    auto gwait = [&](const uint64_t* bar, uint32_t parity, int code) {
        mbar_wait_reported(smem_u32(bar), parity, p.polls, p.err, code);
        __syncwarp();
    };
    pdl_launch_dependents();
    const int half = p.NT / 2;                       // tokens whose activations this CTA brings in

    if (warp == kDeqWarps) {
        // ------------------------------------------------------------------ weight producer
        const int nchunks = p.K / kChunkK, nblocks = (p.N + 63) / 64;
        if (LAYOUT != W_TILED) pdl_wait();           // (the kernel before this one may have written the weights; re-laid-out ones it has not)
        uint32_t slot = 0, ph = 1;
        bool lap = false;
        for (int item = first_item; item < nitems; item += step) {
            const PItem g = p_item(p, item);
            const int b0 = DUAL ? g.row_item * 2 + (int)rank : g.row_item * 4 + (int)rank * 2, b1 = DUAL ? b0 : b0 + 1;     // 64-row blocks
            const unsigned char* w0 = p.w[0] + ((size_t)min(b0, nblocks - 1) * nchunks + g.c_begin) * kRunBytes;
            const unsigned char* w1 = p.w[DUAL ? 1 : 0] + ((size_t)min(b1, nblocks - 1) * nchunks + g.c_begin) * kRunBytes;
#pragma unroll 1
            for (int c = 0; c < g.nc; c++) {
                if (lap) gwait(wempty + slot, ph, 1);
                __syncwarp();
                if (elect_one()) {
                    const uint32_t bar = smem_u32(wfull + slot), dst = smem_u32(ring + G::W0 + slot * G::WSTAGE);
                    if (LAYOUT == W_TILED) {
                        mbar_expect_tx(bar, kTileW);
                        bulk_copy_g2s(dst, w0 + (size_t)c * kRunBytes, kRunBytes, bar);
                        bulk_copy_g2s(dst + kRunBytes, w1 + (size_t)c * kRunBytes, kRunBytes, bar);
                    } else {
                        mbar_expect_tx(bar, LAYOUT == W_BOXES ? G::WSTAGE : 8192);
                        tma_box(dst, &p.wmap, (g.c_begin + c) * 16, b0 * 64, bar);
                        if (LAYOUT == W_BOXES) {
                            tma_box(dst + 8192, &p.smap, (g.c_begin + c) / 4 * 8, b0 * 64, bar);
                            tma_box(dst + 8192 + kTileRows * 16, &p.bmap, (g.c_begin + c) / 4 * 8, b0 * 64, bar);
                        }
                    }
                }
                __syncwarp();
                if (++slot == (uint32_t)G::NW) { slot = 0; ph ^= 1; lap = true; }
            }
        }
    } else if (warp == kDeqWarps + 1) {
        // ------------------------------------------------------------------ activation producer
        const uint32_t xbytes = (uint32_t)half * kChunkK * 2;
        pdl_wait();
        uint32_t slot = 0, ph = 1;
        bool lap = false;
        for (int item = first_item; item < nitems; item += step) {
            const PItem g = p_item(p, item);
            const int tok = g.tok0 + (int)rank * half;
#pragma unroll 1
            for (int c = 0; c < g.nc; c++) {
                if (lap) gwait(xempty + slot, ph, 1);
                __syncwarp();
                if (elect_one()) {
                    const uint32_t bar = smem_u32(xfull + slot), dst = smem_u32(ring + slot * G::X);
                    mbar_expect_tx(bar, xbytes);
                    tma_box(dst, &p.xmap, (g.c_begin + c) * kChunkK, tok, bar);
                    tma_box(dst + half * 128, &p.xmap, (g.c_begin + c) * kChunkK + 64, tok, bar);
                }
                __syncwarp();
                if (++slot == (uint32_t)G::NX) { slot = 0; ph ^= 1; lap = true; }
            }
        }
    } else if (warp == kDeqWarps + 2) {
        uint32_t slot = 0, xph = 0;
        if (rank != 0) {
            // -------------------------------------------------------------- odd CTA: passes on that its activations are there
            for (int item = first_item; item < nitems; item += step) {
                const int nc = p_item(p, item).nc;
#pragma unroll 1
                for (int c = 0; c < nc; c++) {
                    gwait(xfull + slot, xph, 2);
                    if (elect_one()) arrive_pair(peer_addr(smem_u32(xpeer + slot), 0));
                    __syncwarp();
                    if (++slot == (uint32_t)G::NX) { slot = 0; xph ^= 1; }
                }
            }
        } else {
            // -------------------------------------------------------------- MMA issuer (an elected thread of the even CTA)
            const uint32_t idesc = (1u << 4) | ((uint32_t)(p.NT >> 3) << 17) | ((uint32_t)(2 * kTileRows >> 4) << 24);
            const uint64_t xdesc = sw128_desc(smem_u32(ring));
            const uint32_t box = (uint32_t)half * 128 / 16;                              // from one 64-k box to the next, in 16 bytes
            uint32_t ts = 0, tph = 0, it = 0;
            for (int item = first_item; item < nitems; item += step, it++) {
                const PItem g = p_item(p, item);
                if (it > 0) {
                    mbar_wait_reported(smem_u32(&accempty), (it - 1) & 1u, p.polls, p.err, 2);
                    __syncwarp();
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t d0 = tmem + kAcc0;
#pragma unroll 1
                for (int c = 0; c < g.nc; c++) {
                    mbar_wait_reported(smem_u32(xfull + slot), xph, p.polls, p.err, 2);
                    mbar_wait_reported(smem_u32(xpeer + slot), xph, p.polls, p.err, 2);
                    mbar_wait_reported(smem_u32(tready + ts), tph, p.polls, p.err, 2);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (elect_one()) {
                        const uint64_t b0 = xdesc + slot * (G::X / 16);
                        const uint32_t a0 = tmem + ts * kTileCols;
#pragma unroll
                        for (int ks = 0; ks < kChunkK / 16; ks++)
                            asm volatile(
                                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d0),
                                "r"(a0 + ks * 8), "l"(b0 + (ks >> 2) * box + (ks & 3) * 2), "r"(idesc), "r"(ks == 0 ? c : 1)
                                : "memory");
                        commit_to_pair(smem_u32(tfree + ts));
                        commit_to_pair(smem_u32(xempty + slot));
                        if (c == g.nc - 1) commit_to_pair(smem_u32(&accfull));
                    }
                    __syncwarp();
                    if (++slot == (uint32_t)G::NX) { slot = 0; xph ^= 1; }
                    if (++ts == (uint32_t)kGroups) { ts = 0; tph ^= 1; }
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ dequant warps + epilogue
        const int q = warp & 3;
        const uint32_t grp = warp >> 2;                   // takes the chunks with number % 4 == grp, into tensor-memory tile grp; column group in the epilogue
        const int r = q * 32 + lane;                      // weight row inside the tile = tensor-memory lane
        const int rr = r & 15;
        const uint32_t rowoff = LAYOUT == W_TILED ? ((r >> 6) * kRunBytes + ((r >> 4) & 3) * kRecBytes + (rr >> 3) * 512 + (rr & 7) * 64) : r * 64;
        const uint32_t scoff = (r >> 6) * kRunBytes + ((r >> 4) & 3) * kRecBytes + 1024 + rr * 8;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        const uint32_t trow = tmem + grp * kTileCols + lanes;
        const uint32_t ready = peer_addr(smem_u32(tready + grp), 0), drained = peer_addr(smem_u32(&accempty), 0);
        const bool second = DUAL && r >= 64;              // this thread's row is an up row
        const int units = p.NT / 16;                      // of 16 token columns; a column group takes grp, grp + 4, ...
        // first row of this warp's in y (gate / up: of the 64 rows both halves of the tile stand for)
        auto first_row = [&](const PItem& g) { return DUAL ? (g.row_item * 2 + (int)rank) * 64 + (q & 1) * 32 : (g.row_item * 2 + (int)rank) * kTileRows + q * 32; };

        uint32_t sb_s = 0, sb_b = 0;                      // row-major layout: this row's scales and biases of a chunk, loaded one chunk ahead
        auto load_sb = [&](const PItem& g, int c) {
            const size_t e = (size_t)min(first_row(g) + lane, p.N - 1) * (p.K / 64) + (g.c_begin + c) * 2;
            const __half *sp = p.sc + e, *bp = p.bi + e;
            if (p.sb_pairs) {
                sb_s = __ldg(reinterpret_cast<const uint32_t*>(sp));
                sb_b = __ldg(reinterpret_cast<const uint32_t*>(bp));
            } else {
                const unsigned short *su = reinterpret_cast<const unsigned short*>(sp), *bu = reinterpret_cast<const unsigned short*>(bp);
                sb_s = __ldg(su) | (uint32_t)__ldg(su + 1) << 16;
                sb_b = __ldg(bu) | (uint32_t)__ldg(bu + 1) << 16;
            }
        };
        uint32_t it = 0, swaps = 0;
        bool pending = false;
        int prev = 0;

        // Two tokens' products of this lane's row, of token c in the low half -> rows (row & ~1, + 1) of token c + (lane & 1): four bytes
        // a lane to store, two tokens a warp.
        auto across = [&](uint32_t v) {
            const uint32_t w = __shfl_xor_sync(0xffffffffu, v, 1);
            return (lane & 1) ? __byte_perm(w, v, 0x7632) : __byte_perm(v, w, 0x5410);
        };
        // eight packed pairs (tokens tok0 ..) of a unit, after everything but bias and residual
        auto store = [&](const uint32_t* v, int n, int tok0, int row0) {
            const int row = row0 + (lane & ~1), left = row < p.N ? p.M - tok0 - (lane & 1) : 0;      // (N is even)
            const __half2 bv = p.bias != nullptr && left > 0 ? *reinterpret_cast<const __half2*>(p.bias + row) : __float2half2_rn(0.f);
            const bool resid = p.epilogue == B200_EPI_RESIDUAL;
            const size_t at = (size_t)(tok0 + (lane & 1)) * p.N + row, step = 2 * (size_t)p.N;
            __half* dst = p.y + at;
            const __half* src = p.extra + at;
#pragma unroll
            for (int j = 0; j < n; j += 4) {
                uint32_t rs[4];
#pragma unroll
                for (int i = 0; i < 4; i++, src += step) rs[i] = resid && 2 * (j + i) < left ? __ldcg(reinterpret_cast<const unsigned*>(src)) : 0u;
#pragma unroll
                for (int i = 0; i < 4; i++, dst += step) {
                    __half2 o = u32_as_h2(across(v[j + i]));
                    if (p.bias != nullptr) o = __hadd2(o, bv);
                    if (resid) o = __hadd2(u32_as_h2(rs[i]), o);
                    if (2 * (j + i) < left) *reinterpret_cast<__half2*>(dst) = o;
                }
            }
        };
        // a unit's 16 products, rounded and packed
        auto finish = [&](const uint32_t (&h)[8], int unit, const PItem& g) {
            const int tok0 = g.tok0 + unit * 16;
            if (!DUAL) {
                store(h, 8, tok0, first_row(g));
                return;
            }
            // The gate and the up rows of the same outputs stand in warps q and q + 2: each takes half of the tokens and hands over
            // the other half (two buffers in turn, so that one barrier a unit is enough).
            unsigned char* mine = ring + G::SWAP + ((swaps & 1) * kDeqWarps + warp) * 512 + lane * 16;
            const unsigned char* theirs = ring + G::SWAP + ((swaps & 1) * kDeqWarps + (warp ^ 2)) * 512 + lane * 16;
            swaps++;
            *reinterpret_cast<uint4*>(mine) = second ? make_uint4(h[0], h[1], h[2], h[3]) : make_uint4(h[4], h[5], h[6], h[7]);
            asm volatile("bar.sync %0, 64;\n" ::"r"(2 + grp * 2 + (q & 1)) : "memory");
            const uint4 o4 = *reinterpret_cast<const uint4*>(theirs);
            const uint32_t other[4] = {o4.x, o4.y, o4.z, o4.w};
            uint32_t v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t own = second ? h[4 + i] : h[i];
                const float2 gt = __half22float2(u32_as_h2(second ? other[i] : own)), up = __half22float2(u32_as_h2(second ? own : other[i]));
                v[i] = h2_as_u32(__floats2half2_rn(silu_mul_f16(gt.x, up.x), silu_mul_f16(gt.y, up.y)));
            }
            store(v, 4, tok0 + (second ? 8 : 0), first_row(g));
        };
        auto pack = [&](const float (&a)[16], uint32_t (&h)[8]) {
#pragma unroll
            for (int i = 0; i < 8; i++) h[i] = h2_as_u32(__floats2half2_rn(a[2 * i], a[2 * i + 1]));
        };
        auto load_acc = [&](int unit, float (&a)[16]) {
            uint32_t x[16];
            tmem_ld<16>(x, tmem + kAcc0 + lanes + unit * 16);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; i++) a[i] = __uint_as_float(x[i]);
        };
        auto release = [&]() {                            // accumulators read: the next item's MMAs may start
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_pair(drained);
        };
        auto epilogue = [&]() {
            const PItem g = p_item(p, prev);
            gwait(&accfull, (it - 1) & 1u, 3);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            pending = false;
            if (p.splits > 1) {
                // ---- partial products out, four tokens a store: 512 consecutive bytes a warp
                const size_t pstride = (size_t)p.row_items * p.tok_items * 2 * p.NT * (kTileRows / 4);
                float4* const part = reinterpret_cast<float4*>(p.partial) + ((size_t)g.tile * 2 + rank) * p.NT * (kTileRows / 4) + r;
#pragma unroll 1
                for (int unit = grp; unit < units && g.tok0 + unit * 16 < p.M; unit += 4) {
                    float a[16];
                    load_acc(unit, a);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        __stcg(part + g.split * pstride + (unit * 4 + i) * kTileRows, make_float4(a[4 * i], a[4 * i + 1], a[4 * i + 2], a[4 * i + 3]));
                }
                release();
                consumer_sync(kDeqWarps * 32);
                if (threadIdx.x == 0) {
                    int* ctr = p.counter + g.tile * 2 + rank;
                    __threadfence();                      // (with what the block's other threads stored before the barrier)
                    const int old = atomicAdd(ctr, 1);
                    s_last = old == p.splits - 1;
                    if (old == p.splits - 1) *ctr = 0;
                    __threadfence();
                }
                consumer_sync(kDeqWarps * 32);
                const bool last = s_last;
                consumer_sync(kDeqWarps * 32);            // read by all before the next item rewrites it
                if (!last) return;
#pragma unroll 1
                for (int unit = grp; unit < units && g.tok0 + unit * 16 < p.M; unit += 4) {
                    const float4* src = part + (unit * 4) * kTileRows;
                    float4 a[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) a[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                    for (int s = 0; s < p.splits; s += 2) {   // in split order, two of them in flight
                        float4 b[2][4];
#pragma unroll
                        for (int j = 0; j < 2; j++)
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                b[j][i] = s + j < p.splits ? __ldcg(src + (s + j) * pstride + i * kTileRows) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int j = 0; j < 2; j++)
#pragma unroll
                            for (int i = 0; i < 4; i++) { a[i].x += b[j][i].x; a[i].y += b[j][i].y; a[i].z += b[j][i].z; a[i].w += b[j][i].w; }
                    }
                    uint32_t h[8];
                    pack(reinterpret_cast<const float(&)[16]>(a), h);
                    finish(h, unit, g);
                }
                return;
            }
            uint32_t keep[4][8];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if ((int)grp + 4 * u < units) {
                    float a[16];
                    load_acc((int)grp + 4 * u, a);
                    pack(a, keep[u]);
                }
            release();
#pragma unroll
            for (int u = 0; u < 4; u++)
                if ((int)grp + 4 * u < units && g.tok0 + ((int)grp + 4 * u) * 16 < p.M) finish(keep[u], (int)grp + 4 * u, g);
        };

        if (LAYOUT == W_ROWS) pdl_wait();                 // (the kernel before this one may have written the scales)
        uint32_t cbase = 0;                               // chunks of earlier items
        for (int item = first_item;; item += step) {      // once more than there are items, for the last epilogue
            const bool more = item < nitems;
            PItem g{};
            if (more) g = p_item(p, item);
            int k = (int)((grp - cbase) & (kGroups - 1));
            if (LAYOUT == W_ROWS && k < g.nc) load_sb(g, k);
#pragma unroll 1
            do {
                if (k < g.nc) {
                    const uint32_t n = cbase + k, slot = n % G::NW;
                    gwait(wfull + slot, (n / G::NW) & 1u, 3);
                    if (n >= kGroups) gwait(tfree + grp, (n / kGroups - 1) & 1u, 3);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const unsigned char* tile = ring + G::W0 + slot * G::WSTAGE;
                    uint4 u[4];
                    uint32_t sc2[2], bi2[2];                  // scale, bias of the chunk's two k groups, low halves
                    if (LAYOUT == W_TILED) {
#pragma unroll
                        for (int i = 0; i < 4; i++) u[i] = *reinterpret_cast<const uint4*>(tile + rowoff + i * 16);
                        const uint2 sb = *reinterpret_cast<const uint2*>(tile + scoff);
                        sc2[0] = sb.x; bi2[0] = sb.x >> 16;
                        sc2[1] = sb.y; bi2[1] = sb.y >> 16;
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; i++) u[i] = *reinterpret_cast<const uint4*>(tile + rowoff + ((i ^ ((r >> 1) & 3)) << 4));
                        uint32_t sv = sb_s, bv = sb_b;
                        if (LAYOUT == W_BOXES) {
                            const unsigned char* sb = tile + 8192 + r * 16 + ((g.c_begin + k) & 3) * 4;
                            sv = *reinterpret_cast<const uint32_t*>(sb);
                            bv = *reinterpret_cast<const uint32_t*>(sb + kTileRows * 16);
                        } else if (k + kGroups < g.nc) {
                            load_sb(g, k + kGroups);
                        }
                        sc2[0] = sv; sc2[1] = sv >> 16;
                        bi2[0] = bv; bi2[1] = bv >> 16;
                    }
                    const bool fast = __all_sync(0xffffffffu, fast_scale(sc2[0]) && fast_scale(sc2[1]));
                    expand_row<LAYOUT != W_TILED>(u, sc2, bi2, fast, trow);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(wempty + slot));       // the packs have been used
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_pair(ready);
                    k += kGroups;
                }
                // the item before this one: its epilogue runs once this warp's first chunk of this item is expanded
                if (pending) epilogue();
            } while (k < g.nc);
            if (!more) break;
            cbase += g.nc;
            prev = item;
            pending = true;
            it++;
            if (it == 1) pdl_wait();                      // before this thread's first access to what other kernels write
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cluster_arrive();                                // nothing arrives at a CTA that has left; the pair gives its tensor memory back together
    cluster_wait();
    if (warp == kDeqWarps + 2) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
    }
}

template <bool DUAL, int LAYOUT>
int launch_pair(const PairParams& p, int pairs, cudaStream_t stream) {
    auto kern = qmm_pair_kernel<DUAL, LAYOUT>;
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(kern, PGeo<DUAL, LAYOUT>::SMEM, done)) return check_launch();
    const int nitems = p.row_items * p.tok_items * p.splits;
    launch_kernel(kern, dim3(2 * std::min(nitems, pairs)), dim3(kThreads), (size_t)PGeo<DUAL, LAYOUT>::SMEM, stream, p);
    return check_launch();
}

}  // namespace

int qmm_pair(const GemmArgs& a, const PairPlan& pl, cudaStream_t stream) {
    const bool dual = a.epilogue == B200_EPI_SILU_MUL, tiled = a.w_tiled != nullptr;
    PairParams p{};
    int rc = make_map_2d(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, (uint64_t)a.K, (uint64_t)a.M, (uint64_t)a.K * 2, 64, (uint32_t)pl.NT / 2,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200_OK) return rc;
    p.w[0] = static_cast<const unsigned char*>(a.w_tiled);
    p.w[1] = static_cast<const unsigned char*>(a.w2_tiled);
    bool boxes = false;
    if (!tiled) {
        rc = make_map_2d(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, a.wq[0], (uint64_t)a.K / 8, (uint64_t)a.N, (uint64_t)a.K / 2, 16, kTileRows,
                         CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (rc != B200_OK) return rc;
        p.sc = static_cast<const __half*>(a.scales[0]);
        p.bi = static_cast<const __half*>(a.biases[0]);
        p.sb_pairs = ((reinterpret_cast<uintptr_t>(p.sc) | reinterpret_cast<uintptr_t>(p.bi)) & 3u) == 0;
        boxes = a.K % 512 == 0 && aligned16(p.sc) && aligned16(p.bi);
        for (int i = 0; boxes && i < 2; i++) {
            rc = make_map_2d(i ? &p.bmap : &p.smap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, i ? p.bi : p.sc, (uint64_t)a.K / 64, (uint64_t)a.N, (uint64_t)a.K / 32, 8,
                             kTileRows, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
            if (rc != B200_OK) return rc;
        }
    }
    p.bias = static_cast<const __half*>(a.bias);
    p.extra = static_cast<const __half*>(a.extra);
    p.y = static_cast<__half*>(a.y);
    p.counter = a.counters;
    p.err = a.err;
    p.polls = a.err != nullptr ? wait_polls(kWaitPolls, kFirmPolls / 2) : kNoReport;
    p.partial = static_cast<float*>(a.partial);
    p.M = a.M; p.N = a.N; p.K = a.K; p.NT = pl.NT;
    p.row_items = pl.row_items; p.tok_items = pl.tok_items; p.splits = pl.splits; p.chunks_per_split = pl.cps;
    p.epilogue = a.epilogue;
    const int pairs = std::max(1, gemm_sms() / 2);
    if (tiled) return dual ? launch_pair<true, W_TILED>(p, pairs, stream) : launch_pair<false, W_TILED>(p, pairs, stream);
    return boxes ? launch_pair<false, W_BOXES>(p, pairs, stream) : launch_pair<false, W_ROWS>(p, pairs, stream);
}

}  // namespace b200
