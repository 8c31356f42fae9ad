// One forward pass of the 4-bit decoder for up to 32 tokens as a chain of five kernels per layer (programmatic dependent
// launch; the whole step is replayed from a CUDA graph):
//
//   embedding | per layer  A  q|k|v matmul (+ bias), RoPE, KV append      B  tree-masked attention
//                          C  o_proj matmul + residual                    D  gate / up matmul, SiLU(gate) * up
//                          E  down_proj matmul + residual                 | vocabulary projection
//
// Why a chain and not one persistent kernel: a kernel of such a chain whose every CTA reads what all CTAs of its predecessor
// wrote costs 1.0 to 1.3 us, the load included; a device-wide barrier of 148 CTAs took 1.5 to 2.3 us and the first loads behind it
// another 1.1.  A CTA here keeps to half of an SM (512 threads, 64 registers each, ~95 KB of shared memory, 256 columns of tensor memory), so
// the next kernel's CTAs become resident beside it and stream and expand their first weights before its results are there.
//
// RMSNorm is folded into the matmuls around it: the producer of h (embedding, C, E) also writes h * w_norm (fp16, one
// rounding) and sums of h^2 per 32 columns; the consumer multiplies its fp32 accumulator by rsqrt(mean(h^2) + eps).
// All other rounding points are those of the per-op kernels.
//
// Replaces Model.__call__ (mlx_llama.py:298-313) for <= 32 tokens.  Every wait is bounded; one that runs out sets the error
// word of the workspace and the kernel runs to its end.  No copy uses cluster multicast.
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "decode.cuh"
#include "flash.cuh"
#include "pipeline.cuh"
#include "qmm_common.cuh"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace b200 {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kGroups = 3;                       // groups of four dequant warps, each with a tensor-memory tile of its own
constexpr int kDeq = 4 * kGroups;                // dequant warps
constexpr int kEpi = 8;                          // of which these run the epilogue
constexpr int kDThreads = (kDeq + 4) * 32;       // + weight producer, activation producer, MMA issuer, sums of squares
constexpr int kTmem = 256;                       // columns a CTA takes: two CTAs share an SM
constexpr int kMaxCluster = 8;
constexpr int kSsqPitch = 32, kSsqCols = 32, kKeyBlock = 64;

enum { D_QKV = 0, D_RESID = 1, D_SILU = 2, D_HEAD = 3, D_PLAIN = 4, D_ROWS = 5 };      // the last two: y = x W^T (+ bias), a matmul on its own; D_ROWS: W as quantised

template <int TQ>
struct __align__(TQ * 4) Vec { float v[TQ]; };      // a value per token of a group

template <int NT, int TQ = 4>
struct DGeo {
    static constexpr int X = NT * kChunkK * 2;                  // activations of a chunk: two boxes of 64 k
    static constexpr int ACC = kGroups * kTileCols;                  // accumulator columns: two of NT
    static constexpr int NW = 2 * kGroups;                       // weight stages (a multiple: a stage belongs to one of the groups)
    static constexpr int NX = NT == 16 ? 6 : 3;                  // activation stages
    static constexpr int XOFF = NW * kTileW;
    // Partial products [source rank][group of TQ tokens of this CTA][row][TQ] fp32.  The groups go to the CTAs in turn, so at most 8
    // (of four tokens, up to 16), 14 (up to 32: 8 over 7 CTAs) or 8 (of two, up to 8) of them with their sources are here.
    static constexpr int INBOX = XOFF + NX * X;
    static constexpr int SMEM = INBOX + (NT == 16 ? 8 : 14) * kTileRows * TQ * 4 + 1024;
    static_assert(XOFF % 1024 == 0 && 2 * (SMEM + 3072) <= 227 * 1024 && ACC + 2 * NT <= kTmem, "two CTAs per SM");
};

struct DenseParams {
    CUtensorMap xmap;             // activations [M][K], boxes of 64 k x NT rows, 128-byte swizzle
    const unsigned char* w[2];    // streaming layout (gate / up)
    const __half* bias;
    const __half* wn;             // norm weights applied to the new h (D_RESID)
    __half* y;                    // q|k|v, activations or logits
    __half* h;                    // residual stream (D_RESID)
    __half* hw;
    float* ssq;                   // [H / 32][32]
    int H;
    float eps;
    int M, N, K;                  // N: output rows of each matrix
    int tile_lo, tiles;           // 128-row tiles (64 + 64 rows of gate and up): first and end
    int* err;
    int polls;                    // of a wait before it gives up
    // D_QKV
    const float2* cs;             // [token][hd / 2] (cos, sin)
    __half* kc;                   // this layer's K and V of request 0
    __half* vc;
    const int* prefix;
    int Hq, Hkv, hd, cap, write_off, mr;      // WIDE: write_off is the first cache row of the pass
    size_t req_stride;            // halves between the caches of two requests
    // D_ROWS: packs [N][K / 8] as rows of bytes, boxes of 64 bytes x 128 rows, 64-byte swizzle; scales and biases [N][K / 64]
    CUtensorMap wmap;
    union {
        const __half* sc;
        const void* const* tw;    // TABLE: weights (gate, then up) in a layer table in device memory, for callers without a copy of it on the host
    };
    union {
        const __half* bi;
        const void* const* tv;    // TABLE: bias (D_QKV), norm weights (D_RESID) there; NULL: as given above
    };
    // D_HEAD
    const int* row_index;
    int rows_out;
};
template <typename T>
__device__ __forceinline__ const T* listed(const void* const* entry) {
    return reinterpret_cast<const T*>(__ldcg(reinterpret_cast<const unsigned long long*>(entry)));
}

template <int TQ>
__device__ __forceinline__ void st_async(uint32_t addr, const uint32_t* a, uint32_t bar) {
    if (TQ == 4)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(addr), "r"(a[0]), "r"(a[1]),
                     "r"(a[TQ - 2]), "r"(a[TQ - 1]), "r"(bar) : "memory");
    else
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];\n" ::"r"(addr), "r"(a[0]), "r"(a[1]), "r"(bar) : "memory");
}
// ================================================================================ matmul kernel
// Grid: 128-row tiles x cluster ranks; the cluster's CTAs share a tile's K range.  Each finishes its share of the token
// columns: the others store their fp32 partial products for it straight into its shared memory and arrive at its barrier (a
// cluster barrier and reading them from there took 1 us more).
//
// Three groups of four dequant warps (thread = weight row) take the chunks in turn, each with a tensor-memory tile; one MMA warp
// follows in order.  Three chunks are expanded before the wait for the previous kernel: behind it
// come the activation load (0.5 us), the MMAs (0.1 us a chunk) and the epilogue.  Code that runs once per kernel is kept short:
// cold instructions cost 2 to 4 cycles each.
// WIDE (prompts): blockIdx.y counts tiles of NT tokens, each with CTAs of its own that stream and expand the weights for themselves.  The input
// is normed already, in fp32 by a kernel of its own as in longer prompts: h * w_norm before 1 / rms, in fp16, has less of a range.
// FAST: every scale is known to allow the short expansion (b200_forward_desc.scales_in_fast_range).  Asking every chunk, with the long
// expansion at hand, made the 18944 x 3584 pair 18.6 us and not 17.7, the vocabulary projection of the 7B shape 74 and not 68.
template <int NT, int KIND, int TQ, bool TABLE = false, bool WIDE = false, bool FAST = false>
__global__ void __launch_bounds__(kDThreads, 2) dense_kernel(const __grid_constant__ DenseParams p) {
    using G = DGeo<NT, TQ>;
    using V = Vec<TQ>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    V* inbox = reinterpret_cast<V*>(ring + G::INBOX);
    __shared__ uint64_t wfull[G::NW], wempty[G::NW], xfull[G::NX], xempty[G::NX], tready[kGroups], tfree[kGroups], accfull[2], accempty[2], inboxfull;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(16) float s_rs[32];                                   // 1 / rms per token
    __shared__ int s_base[32];                                                 // per request: committed rows (D_QKV), first row of logits (D_HEAD)

    constexpr bool NORMED = !WIDE && KIND != D_RESID && KIND != D_PLAIN && KIND != D_ROWS;               // the input is h * w_norm: scale by 1 / rms
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank(), cs = cluster_size();
    const int tile0 = p.tile_lo + blockIdx.x / (int)cs, tstep = gridDim.x / (int)cs;
    const int nit = cs > 1 ? 1 : (p.tiles - tile0 + tstep - 1) / tstep;                                   // this CTA's tiles: tile0, + tstep, ...
    const int nchunks = p.K / kChunkK;
    const int c_lo = nchunks * (int)rank / (int)cs, nc = nchunks * ((int)rank + 1) / (int)cs - c_lo;      // chunks of each
    const int t0 = WIDE ? (int)blockIdx.y * NT : 0, M = WIDE ? min(NT, p.M - t0) : p.M, mr = WIDE ? M : p.mr;       // first token, tokens, of a request
    const int quads = (M + TQ - 1) / TQ, qslots = (quads + (int)cs - 1) / (int)cs;                      // groups of tokens, most of a CTA's
    const int nq = quads > (int)rank ? (quads - (int)rank + (int)cs - 1) / (int)cs : 0;                   // this CTA finishes rank, rank + cs, ...

    if (threadIdx.x < 32) {                                      // (a thread a barrier: one thread for all took 400 cycles)
        if (lane < G::NX) {
            mbar_init(smem_u32(xfull + lane), 1);
            mbar_init(smem_u32(xempty + lane), 1);
        }
        if (lane < kGroups) {
            mbar_init(smem_u32(tready + lane), 4);
            mbar_init(smem_u32(tfree + lane), 1);
        }
        if (lane < 2) {
            mbar_init(smem_u32(accfull + lane), 1);
            mbar_init(smem_u32(accempty + lane), kEpi);
        }
        if (lane == 31) {
            mbar_init(smem_u32(&inboxfull), 1);
            if (cs > 1) mbar_expect_tx(smem_u32(&inboxfull), cs * nq * kTileRows * TQ * 4); // what the cluster's CTAs will store here
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    // The weight producer makes its own barriers and asks for the first stages before the block is set up.
    const int nblocks = (p.N + 63) / 64;
    auto wsrc = [&](int tile, int second) {                      // chunk c_lo of the tile's first or second 64 rows (gate / up: of the same rows of each)
        const unsigned char* w = TABLE ? listed<unsigned char>(p.tw + (KIND == D_SILU ? second : 0)) : p.w[KIND == D_SILU ? second : 0];
        return w + ((size_t)(KIND == D_SILU ? tile : min(2 * tile + second, nblocks - 1)) * nchunks + c_lo) * kRunBytes;
    };
    auto wload = [&](uint32_t slot, const unsigned char* src0, const unsigned char* src1) {
        const uint32_t bar = smem_u32(wfull + slot), dst = smem_u32(ring + slot * kTileW);
        mbar_expect_tx(bar, kTileW);
        bulk_copy_g2s(dst, src0, kRunBytes, bar);
        bulk_copy_g2s(dst + kRunBytes, src1, kRunBytes, bar);
    };
    auto wload_rows = [&](uint32_t slot, int tile, int c) {
        const uint32_t bar = smem_u32(wfull + slot);
        mbar_expect_tx(bar, kTileRows * 64);
        tma_box(smem_u32(ring + slot * kTileW), &p.wmap, (c_lo + c) * 64, tile * kTileRows, bar);
    };
    if (warp == kDeq) {
        if (lane < G::NW) {
            mbar_init(smem_u32(wfull + lane), 1);
            mbar_init(smem_u32(wempty + lane), 4);               // a group's warps
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
        if (KIND == D_ROWS) pdl_wait();                          // (the kernel before this one may have written the weights)
        if (elect_one()) {
            const unsigned char *src0 = wsrc(tile0, 0), *src1 = wsrc(tile0, 1);
#pragma unroll 1
            for (int c = 0; c < min(nc, G::NW); c++) {
                if (KIND == D_ROWS) wload_rows(c, tile0, c);
                else wload(c, src0 + c * kRunBytes, src1 + c * kRunBytes);
            }
        }
        __syncwarp();
    }
    if (warp == kDeq + 1 && lane == 0) asm volatile("prefetch.tensormap [%0];\n" ::"l"(&p.xmap) : "memory");
    if (warp == kDeq + 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "n"(kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();
    if (cs > 1) cluster_arrive_relaxed();                        // (waited for before the first store to a peer)

    if (warp == kDeq) {
        // ------------------------------------------------------------------ weight producer: depends on nothing
        const int first = min(nc, G::NW);                        // (asked for above)
        uint32_t slot = first % G::NW, ph = 1;
        bool lap = first == G::NW;
        if (lap) ph = 0;
#pragma unroll 1
        for (int it = 0, tile = tile0; it < nit; it++, tile += tstep) {
            const int c0 = it == 0 ? first : 0;
            const unsigned char *src0 = wsrc(tile, 0) + c0 * kRunBytes, *src1 = wsrc(tile, 1) + c0 * kRunBytes;
#pragma unroll 1
            for (int c = c0; c < nc; c++) {
                if (lap) mbar_wait_reported(smem_u32(wempty + slot), ph, p.polls, p.err, 21);
                __syncwarp();
                if (elect_one()) {
                    if (KIND == D_ROWS) wload_rows(slot, tile, c);
                    else wload(slot, src0, src1);
                }
                __syncwarp();
                src0 += kRunBytes;
                src1 += kRunBytes;
                if (++slot == (uint32_t)G::NW) { slot = 0; ph ^= 1; lap = true; }
            }
        }
    } else if (warp == kDeq + 1) {
        // ------------------------------------------------------------------ activation producer
        pdl_wait();
        uint32_t slot = 0, ph = 1;
        bool lap = false;
        for (int it = 0; it < nit; it++)
#pragma unroll 1
            for (int c = 0; c < nc; c++) {
                if (lap) mbar_wait_reported(smem_u32(xempty + slot), ph, p.polls, p.err, 26);
                __syncwarp();
                if (elect_one()) {
                    const uint32_t bar = smem_u32(xfull + slot), dst = smem_u32(ring + G::XOFF + slot * G::X);
                    mbar_expect_tx(bar, G::X);
                    tma_box(dst, &p.xmap, (c_lo + c) * kChunkK, t0, bar);
                    tma_box(dst + NT * 128, &p.xmap, (c_lo + c) * kChunkK + 64, t0, bar);
                }
                __syncwarp();
                if (++slot == (uint32_t)G::NX) { slot = 0; ph ^= 1; lap = true; }
            }
    } else if (warp == kDeq + 2) {
        // ------------------------------------------------------------------ MMA issuer (an elected thread)
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
        const uint64_t xdesc = sw128_desc(smem_u32(ring + G::XOFF));
        uint32_t tl = 0, tph = 0, slot = 0, xph = 0;
#pragma unroll 1
        for (int it = 0; it < nit; it++) {
            const uint32_t ab = it & 1, d0 = tmem + G::ACC + ab * NT;
            if (it >= 2) mbar_wait_reported(smem_u32(accempty + ab), ((it >> 1) - 1) & 1, p.polls, p.err, 27);
#pragma unroll 1
            for (int c = 0; c < nc; c++) {
                mbar_wait_reported(smem_u32(xfull + slot), xph, p.polls, p.err, 22);
                mbar_wait_reported(smem_u32(tready + tl), tph, p.polls, p.err, 22);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (elect_one()) {                               // (~285 cycles a batch; of half the size, 280)
                    const uint64_t b0 = xdesc + slot * (G::X / 16);
                    const uint32_t a0 = tmem + tl * kTileCols;
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d0),
                                 "r"(a0), "l"(b0), "r"(idesc), "r"(c) : "memory");
#pragma unroll
                    for (int ks = 1; ks < kChunkK / 16; ks++)
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d0),
                                     "r"(a0 + ks * 8), "l"(b0 + ((ks >> 2) * (NT * 128) + (ks & 3) * 32) / 16), "r"(idesc) : "memory");
                    commit_to(smem_u32(tfree + tl));
                    commit_to(smem_u32(xempty + slot));
                    if (c == nc - 1) commit_to(smem_u32(accfull + ab));
                }
                __syncwarp();
                if (++tl == (uint32_t)kGroups) { tl = 0; tph ^= 1; }
                if (++slot == (uint32_t)G::NX) { slot = 0; xph ^= 1; }
            }
        }
        asm volatile("bar.sync 2, %0;\n" ::"n"((kEpi + 1) * 32) : "memory");         // accumulators read
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(kTmem) : "memory");
    } else if (warp == kDeq + 3) {
        // ------------------------------------------------------------------ sums of squares -> 1 / rms of each token
        // (by the dequant warps it held up every chunk behind the first three: 1.4 us at a hidden size of 3584)
        // The epilogue's parameters are asked for ahead of the wait: read for the first time behind it, each line is a miss on the way.
        asm volatile("" ::"l"(p.bias), "l"(p.wn), "l"(p.y), "l"(p.h), "l"(p.hw), "l"(p.ssq), "r"(p.H), "f"(p.eps), "r"(p.M), "r"(p.N), "r"(p.tiles), "l"(p.err), "r"(p.polls));
        if (KIND == D_QKV)
            asm volatile("" ::"l"(p.cs), "l"(p.kc), "l"(p.vc), "l"(p.prefix), "r"(p.Hq), "r"(p.Hkv), "r"(p.hd), "r"(p.cap), "r"(p.write_off), "r"(p.mr), "l"(p.req_stride));
        if (KIND == D_HEAD) asm volatile("" ::"r"(p.mr), "l"(p.row_index), "r"(p.rows_out));
        if (NORMED) {
            // (both were there before the pass; read in the epilogue they were 0.5 us of every q|k|v kernel)
            if (KIND == D_QKV && lane < M / mr) s_base[lane] = __ldcg(p.prefix + lane);
            if (KIND == D_HEAD && lane < M / mr) s_base[lane] = p.row_index != nullptr ? __ldcg(p.row_index + lane) : 0;
            pdl_wait();
            // A lane: four tokens of every `step`-th part, four or eight loads in flight whatever the number of parts.  (Unrolled by seven with
            // the rest one at a time: 4.3 us at 3584 x 16 tokens and 8.3 at 4096 x 32, longer than the MMAs.  Parts of 128 columns, added up
            // by the producer's warps: 0.15 us more for each of them, of 2.7 in a draft-sized layer.)
            const int parts = p.H / kSsqCols, quads = M <= 8 ? 2 : (M <= 16 ? 4 : 8), step = 32 / quads, quad = lane & (quads - 1);
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            constexpr int FLY = NT == 16 ? 4 : 8;
#pragma unroll 1
            for (int part = lane / quads; part < parts; part += FLY * step) {
                float4 v[FLY];
#pragma unroll
                for (int i = 0; i < FLY; i++)
                    v[i] = part + i * step < parts ? __ldcg(reinterpret_cast<const float4*>(p.ssq + (part + i * step) * kSsqPitch + quad * 4))
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < FLY; i++) { t.x += v[i].x; t.y += v[i].y; t.z += v[i].z; t.w += v[i].w; }
            }
            __syncwarp();
            for (int o = 16; o >= quads; o >>= 1) {
                t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
                t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
                t.z += __shfl_xor_sync(0xffffffffu, t.z, o);
                t.w += __shfl_xor_sync(0xffffffffu, t.w, o);
            }
            if (lane < quads) {
                s_rs[quad * 4] = rsqrtf(t.x / (float)p.H + p.eps);
                s_rs[quad * 4 + 1] = rsqrtf(t.y / (float)p.H + p.eps);
                s_rs[quad * 4 + 2] = rsqrtf(t.z / (float)p.H + p.eps);
                s_rs[quad * 4 + 3] = rsqrtf(t.w / (float)p.H + p.eps);
            }
            __syncwarp();
            asm volatile("bar.arrive 3, %0;\n" ::"n"((kEpi + 1) * 32) : "memory");
        }
    } else {
        // ------------------------------------------------------------------ dequant warps
        const uint32_t me = warp >> 2;                           // group (and, in the epilogue, which half of the tokens)
        const int q = warp & 3, r = q * 32 + lane, rr = r & 15;
        const uint32_t recoff = (r >> 6) * kRunBytes + ((r >> 4) & 3) * kRecBytes;
        const uint32_t rowoff = KIND == D_ROWS ? r * 64 + (((r >> 1) & 3) << 4) : recoff + (rr >> 3) * 512 + (rr & 7) * 64, scoff = recoff + 1024 + rr * 8;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16);
        // (Four threads of a quarter-warp read the same banks: swapping units between threads to halve that took more issue slots, 16
        // selects a chunk, than the reads took cycles.)
        const __half* const wn = TABLE && KIND == D_RESID && p.tv != nullptr ? listed<__half>(p.tv) : p.wn;
        const __half* const bias = TABLE && KIND == D_QKV ? listed<__half>(p.tv) : p.bias;
        // ---- one finished tile: accumulators -> inbox of the CTA that finishes each token -> output
        auto epilogue = [&](int it) {
            const int tile = tile0 + it * tstep;
            const uint32_t ab = it & 1;
            const int r2 = KIND == D_SILU ? threadIdx.x & 63 : threadIdx.x & 127;     // row inside the tile that this thread finishes
            const int j0 = KIND == D_SILU ? threadIdx.x >> 6 : threadIdx.x >> 7;      // its first quad of this CTA's, and the step
            constexpr int JS = KIND == D_SILU ? 4 : 2;
            const int n = (KIND == D_SILU ? tile * 64 : tile * kTileRows) + r2;
            const bool valid = n < p.N;
            // what the output needs besides the product, asked for now: norm weight or bias, the first quad's residuals or rotations
            const int half = p.hd >> 1, hi = r2 & (p.hd - 1), head = KIND == D_QKV ? n >> (p.hd == 128 ? 7 : 6) : 0;
            const bool rotate = KIND == D_QKV && head < p.Hq + p.Hkv, first = hi < half;
            const int pr = rotate ? (first ? r2 + half : r2 - half) : r2;      // the row it is rotated with, inside this tile
            __half extra = __ushort_as_half(0), extra2 = __ushort_as_half(0);
            unsigned short hres[TQ];
            float2 rot[TQ];
            auto ask = [&](int j) {                              // (warp-uniform j and token counts)
                const int tok0 = TQ * ((int)rank + j * (int)cs);
#pragma unroll
                for (int k = 0; k < TQ; k++) {
                    if (KIND == D_RESID && valid && tok0 + k < M)
                        hres[k] = __ldcg(reinterpret_cast<const unsigned short*>(p.h) + (size_t)(t0 + tok0 + k) * p.N + n);
                    if (KIND == D_QKV && rotate && tok0 + k < M) rot[k] = __ldcg(p.cs + (t0 + tok0 + k) * kCsPitch + (first ? hi : hi - half));
                }
            };
            if (it == 0) pdl_wait();
            if (KIND == D_RESID && !WIDE && valid) extra = wn[n];
            if ((KIND == D_QKV || KIND == D_PLAIN || KIND == D_ROWS) && valid && bias != nullptr) {
                extra = bias[n];
                if (KIND == D_QKV) extra2 = bias[tile * kTileRows + pr];
            }
            if (j0 < nq) ask(j0);
            if (cs > 1) cluster_wait();                          // (the peers have started: while the last MMAs run)

            mbar_wait_reported(smem_u32(accfull + ab), (it >> 1) & 1, p.polls, p.err, 23);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            constexpr int C = NT / 2;                            // columns of this warp
            uint32_t a[C];
#pragma unroll
            for (int i = 0; i < C; i += 8)
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                             : "=r"(a[i]), "=r"(a[i + 1]), "=r"(a[i + 2]), "=r"(a[i + 3]), "=r"(a[i + 4]), "=r"(a[i + 5]), "=r"(a[i + 6]), "=r"(a[i + 7])
                             : "r"(tmem + G::ACC + ab * NT + me * C + i + ((uint32_t)(q * 32) << 16)) : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            if (it == nit - 1) asm volatile("bar.arrive 2, %0;\n" ::"n"((kEpi + 1) * 32) : "memory");     // tensor memory may be given back
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(accempty + ab));
            if (cs == 1) {
                if (it > 0) consumer_sync(kEpi * 32);            // the tile before this one has been read
#pragma unroll
                for (int i = 0; i < C; i += TQ)
                    if ((int)me * C + i < M) {
                        V x;
#pragma unroll
                        for (int k = 0; k < TQ; k++) x.v[k] = __uint_as_float(a[i + k]);
                        inbox[((int)me * C + i) / TQ * kTileRows + r] = x;
                    }
                consumer_sync(kEpi * 32);
            } else {
                // A store into a peer's memory counts its bytes at the peer's barrier by itself: no fence, no arrival behind it.  TQ
                // tokens a store: with one, the stores were what a pass of many tokens waited for (1.1 us for four more tokens).
                const uint32_t in0 = smem_u32(inbox), inbar = smem_u32(&inboxfull);
                uint32_t dst = (me * (C / TQ)) % cs, sl = (me * (C / TQ)) / cs;
#pragma unroll
                for (int i = 0; i < C; i += TQ) {
                    if ((int)me * C + i < M)
                        st_async<TQ>(peer_addr(in0 + ((rank * qslots + sl) * kTileRows + r) * (TQ * 4), dst), a + i, peer_addr(inbar, dst));
                    if (++dst == cs) { dst = 0; sl++; }
                }
                inbox_wait(inbar, p.polls, p.err, 28);
                __syncwarp();
            }
            if (NORMED && it == 0) asm volatile("bar.sync 3, %0;\n" ::"n"((kEpi + 1) * 32) : "memory");      // s_rs
#pragma unroll 1
            for (int j = j0; j < nq; j += JS) {                  // (warp-uniform)
                const int tok0 = TQ * ((int)rank + j * (int)cs);
                if (j != j0) ask(j);
                // the sources in rank order: this row, and the up row or the one it is rotated with
                const int r3 = KIND == D_SILU ? r2 + 64 : pr;
                V v = inbox[j * kTileRows + r2], w = v;
                if (KIND == D_SILU || KIND == D_QKV) w = inbox[j * kTileRows + r3];
#pragma unroll 1
                for (int i = 1; i < (int)cs; i++) {
                    const V* src = inbox + (i * qslots + j) * kTileRows;
                    const V x = src[r2];
#pragma unroll
                    for (int k = 0; k < TQ; k++) v.v[k] += x.v[k];
                    if (KIND == D_SILU || KIND == D_QKV) {
                        const V y = src[r3];
#pragma unroll
                        for (int k = 0; k < TQ; k++) w.v[k] += y.v[k];
                    }
                }
                if (NORMED) {
                    const V rs = *reinterpret_cast<const V*>(s_rs + tok0);
#pragma unroll
                    for (int k = 0; k < TQ; k++) { v.v[k] *= rs.v[k]; w.v[k] *= rs.v[k]; }
                }
                float ss[TQ] = {};
#pragma unroll
                for (int k = 0; k < TQ; k++) {
                    const int tok = tok0 + k;
                    if (tok >= M) break;
                    const int rq = KIND == D_HEAD || KIND == D_QKV ? (mr == M ? 0 : tok / mr) : 0;
                    if (KIND == D_SILU) {
                        if (valid) p.y[(size_t)(t0 + tok) * p.N + n] = __float2half_rn(silu_mul_f16(v.v[k], w.v[k]));
                    } else if (KIND == D_RESID) {
                        if (valid) {
                            const size_t at = (size_t)(t0 + tok) * p.N + n;
                            const __half o = __hadd(__ushort_as_half(hres[k]), __float2half_rn(v.v[k]));
                            const float f = __half2float(o);
                            ss[k] = f * f;
                            p.h[at] = o;
                            if (!WIDE) p.hw[at] = __hmul(o, extra);
                        }
                    } else if (KIND == D_PLAIN || KIND == D_ROWS) {
                        __half x = __float2half_rn(v.v[k]);
                        if (bias != nullptr) x = __hadd(x, extra);
                        if (valid) p.y[(size_t)tok * p.N + n] = x;
                    } else if (KIND == D_HEAD) {
                        const int rel = tok - rq * mr - s_base[rq];
                        if (valid && rel >= 0 && rel < p.rows_out) p.y[(size_t)(rq * p.rows_out + rel) * p.N + n] = __float2half_rn(v.v[k]);
                    } else {
                        __half x = __float2half_rn(v.v[k]);
                        if (bias != nullptr) x = __hadd(x, extra);
                        if (rotate) {
                            __half y = __float2half_rn(w.v[k]);
                            if (bias != nullptr) y = __hadd(y, extra2);
                            const float xs = __half2float(x), ys = __half2float(y);
                            x = __float2half_rn(first ? xs * rot[k].x - ys * rot[k].y : ys * rot[k].y + xs * rot[k].x);
                        }
                        if (valid) {
                            if (head < p.Hq) {
                                p.y[(size_t)(t0 + tok) * p.N + n] = x;
                            } else {
                                const int row = (WIDE ? t0 : s_base[rq]) + p.write_off + (tok - rq * mr);
                                const int kvh = head - p.Hq - (rotate ? 0 : p.Hkv);
                                if (row < p.cap) ((rotate ? p.kc : p.vc) + (size_t)rq * p.req_stride)[((size_t)kvh * p.cap + row) * p.hd + hi] = x;
                            }
                        }
                    }
                }
                if (KIND == D_RESID && !WIDE) {
                    // sums over the warp's rows, halving the tokens a lane holds with the first steps: token lane / (32 / TQ) in the end
                    float x = ss[0];
                    if (TQ == 4) {
                        const bool hi = lane & 16, odd = lane & 8;
                        const float x0 = (hi ? ss[TQ - 2] : ss[0]) + __shfl_xor_sync(0xffffffffu, hi ? ss[0] : ss[TQ - 2], 16);
                        const float x1 = (hi ? ss[TQ - 1] : ss[1]) + __shfl_xor_sync(0xffffffffu, hi ? ss[1] : ss[TQ - 1], 16);
                        x = (odd ? x1 : x0) + __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 8);
                    } else {
                        const bool hi = lane & 16;
                        x = (hi ? ss[1] : ss[0]) + __shfl_xor_sync(0xffffffffu, hi ? ss[0] : ss[1], 16);
                    }
#pragma unroll
                    for (int o = 16 / TQ; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if ((lane & (32 / TQ - 1)) == 0 && valid && tok0 + lane / (32 / TQ) < M)
                        p.ssq[(n >> 5) * kSsqPitch + tok0 + lane / (32 / TQ)] = x;
                }
            }
        };
        uint32_t slot = me, wph = 0, tph = 1;
        int done = me;                                           // number of this group's next chunk, over all tiles
        // D_ROWS: scales and biases of the group's next chunk (two groups of 64), asked for a chunk ahead
        uint32_t next_s = 0, next_b = 0;
        int ask_tile = tile0, ask_c = (int)me;
        auto ask_scales = [&]() {
            while (ask_c >= nc && ask_tile < p.tiles) { ask_c -= nc; ask_tile += tstep; }
            if (ask_tile < p.tiles) {
                const size_t at = (size_t)min(ask_tile * kTileRows + r, p.N - 1) * (p.K / 64) + 2 * (c_lo + ask_c);
                next_s = __ldg(reinterpret_cast<const uint32_t*>(p.sc + at));
                next_b = __ldg(reinterpret_cast<const uint32_t*>(p.bi + at));
            }
            ask_c += kGroups;
        };
        if (KIND == D_ROWS) {
            pdl_wait();
            ask_scales();
        }
#pragma unroll 1
        for (int it = 0; it <= nit; it++) {
            const int end = it < nit ? (it + 1) * nc : 0;
            bool pending = it > 0;                               // the tile before this one, once two chunks of this one are expanded:
            int ahead = 0;                                       // its last MMA is done by then
#pragma unroll 1
            do {
                if (done < end) {
                    mbar_wait_reported(smem_u32(wfull + slot), wph, p.polls, p.err, 24);
                    const unsigned char* st = ring + slot * kTileW;
                    uint4 u[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) u[i] = *reinterpret_cast<const uint4*>(st + (KIND == D_ROWS ? rowoff ^ (i * 16) : rowoff + i * 16));
                    uint32_t sc[2], bi[2];                       // scale and bias of the chunk's two groups, low halves
                    if (KIND == D_ROWS) {
                        sc[0] = next_s; sc[1] = next_s >> 16;
                        bi[0] = next_b; bi[1] = next_b >> 16;
                        ask_scales();
                    } else {
                        const uint2 sb = *reinterpret_cast<const uint2*>(st + scoff);
                        sc[0] = sb.x; bi[0] = sb.x >> 16;
                        sc[1] = sb.y; bi[1] = sb.y >> 16;
                    }
                    const bool fast = FAST || __all_sync(0xffffffffu, fast_scale(sc[0]) && fast_scale(sc[1]));
                    if (done >= kGroups) mbar_wait_reported(smem_u32(tfree + me), tph, p.polls, p.err, 24);
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    expand_row<KIND == D_ROWS, KIND == D_PLAIN && NT == 32>(u, sc, bi, fast, trow + me * kTileCols);
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    // The stage is given back only now that the packs have been used: an arrival right behind the loads does not wait for them, and
                    // the next tile's weights were there before the last of them were through (some rows of one stage in 1e8; 46 wrong passes of
                    // 200000).
                    if (lane == 0) {
                        mbar_arrive(smem_u32(tready + me));
                        mbar_arrive(smem_u32(wempty + slot));
                    }
                    done += kGroups;
                    ahead++;
                    if ((slot += kGroups) >= (uint32_t)G::NW) { slot -= G::NW; wph ^= 1; }
                    tph ^= 1;
                }
                if (pending && (ahead == 2 || done >= end)) {
                    if (warp < kEpi) epilogue(it - 1);
                    pending = false;
                }
            } while (done < end);
        }
        if (warp < kEpi) return;
    }
    if (cs > 1) cluster_wait();
}

// ================================================================================ embedding
// One CTA per token: dequantised embedding row -> h, h * w_norm, sums of squares per 32 columns, and the token's RoPE table.  The norm
// weights may come from the layer table (`wn_entry`).
// The next kernel is let go only behind the wait: everything before the pass (tree kernels, KV compaction, other programs'
// writes) is then complete before any kernel of the pass starts, which may so read committed K/V rows, and the layer table, ahead
// of its own wait.
__global__ void __launch_bounds__(256) embed_kernel(const int* __restrict__ tokens, const int* __restrict__ pos, const uint32_t* __restrict__ wq,
                                                    const __half* __restrict__ sc, const __half* __restrict__ bi, const __half* wn,
                                                    __half* __restrict__ h, __half* __restrict__ hw, float* __restrict__ ssq,
                                                    float2* __restrict__ cs, const float* __restrict__ inv_freq, float scaling, int H, int V,
                                                    int half_hd, const void* const* wn_entry) {
    pdl_wait();
    pdl_launch_dependents();
    if (wn_entry != nullptr) wn = listed<__half>(wn_entry);
    const int m = blockIdx.x, units = H / 8;
    const int tok = min(max(tokens[m], 0), V - 1);
    for (int u = threadIdx.x; u < ((units + 31) & ~31); u += 256) {
        float ss = 0.f;
        if (u < units) {
            const uint32_t w = wq[(size_t)tok * units + u];
            const __half s = sc[(size_t)tok * (H / 64) + (u >> 3)], b = bi[(size_t)tok * (H / 64) + (u >> 3)];
            const uint4 wv = *reinterpret_cast<const uint4*>(wn + u * 8);
            const __half* wh = reinterpret_cast<const __half*>(&wv);
            __align__(16) __half o[8], ow[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                o[j] = __hfma(__int2half_rn((int)((w >> (4 * j)) & 0xfu)), s, b);
                const float f = __half2float(o[j]);
                ss += f * f;
                ow[j] = __hmul(o[j], wh[j]);
            }
            *reinterpret_cast<uint4*>(h + (size_t)m * H + u * 8) = *reinterpret_cast<const uint4*>(o);
            *reinterpret_cast<uint4*>(hw + (size_t)m * H + u * 8) = *reinterpret_cast<const uint4*>(ow);
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (u < units && (u & 3) == 0) ssq[(u >> 2) * kSsqPitch + m] = ss;
    }
    if ((int)threadIdx.x < half_hd) {
        float s, c;
        sincosf((scaling * inv_freq[threadIdx.x]) * (float)pos[m], &s, &c);
        cs[m * kCsPitch + threadIdx.x] = make_float2(c, s);
    }
}

// ================================================================================ attention of up to 16 query rows
// (More of them, and long caches at head dim 128: csrc/flash.cu.)
// CTA = (key range, kv head, request); a query row is (token, head of the group).  Four warps share the tile of 16
// rows: each takes a quarter of a block's keys for the scores and, the probabilities exchanged through shared memory, a quarter of the
// dims for the output, so partial outputs leave the CTA once per row.  All share the K/V blocks (TMA boxes, 128-byte swizzle).  The CTAs of a
// cluster take neighbouring key ranges; each finishes its share of the rows, whose partial softmax states the others store into its shared
// memory, merged in range order.  Committed blocks are asked for before the wait for the kernel that appends this pass's rows.
struct DAttn {
    CUtensorMap kvmap;             // the cache as [rows][head_dim], 64 x 64 boxes
    const __half* q;               // q|k|v buffer [M][pitch], q rotated
    int pitch;
    const unsigned long long* mask;
    const int* prefix;
    __half* out;                   // [M][Hq * HD]
    int Hq, Hkv, mr, tail, nkb;
    int row0, req_rows, cap, write_off;    // cache row of (this layer, K, head 0), rows of one request's cache
    float scale_log2;
    int* err;
    int polls;
};

__device__ __forceinline__ uint32_t kv_swz(int r, int v) {     // 16-byte vector v of row r of a block (boxes of 8 vectors side by side)
    return (uint32_t)((v >> 3) * 8192 + r * 128 + (((v & 7) ^ (r & 7)) << 4));
}
constexpr int kAWarps = 4;                         // warps of an attention CTA: they share a row tile
template <int HD>
struct DAGeo {
    static constexpr int ROWS = 16;                                      // query rows of a CTA
    static constexpr int BLOCK = 2 * 64 * HD * 2;                        // K and V of 64 keys
    static constexpr int STAGES = HD == 128 ? 2 : 3;
    static constexpr int Q = STAGES * BLOCK;                             // queries [row][HD], 16-byte units swizzled
    static constexpr int P = Q + ROWS * HD * 2;                          // probabilities of a block [16][64], swizzled
    static constexpr int OP = HD + 4;                                    // floats per row of a partial output
    static constexpr int INBOX = P + ROWS * 128;                         // partial outputs [source CTA][row of this CTA][OP]
    static constexpr int INBOX_ML = INBOX + (ROWS + kMaxCluster) * OP * 4;       // and (max, sum) [source CTA][part][row]
    static constexpr int SMEM = INBOX_ML + kAWarps * (ROWS + kMaxCluster) * 8 + 1024;
    static_assert(2 * (SMEM + 2048) <= 227 * 1024 && SMEM + DGeo<32>::SMEM + 4 * 1024 <= 227 * 1024, "two CTAs per SM, or one beside a matmul CTA");
};

template <int HD>
__global__ void __launch_bounds__(kAWarps * 32) attention_kernel(const __grid_constant__ DAttn p) {
    using G = DAGeo<HD>;
    constexpr int PT = kAWarps;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    __shared__ uint64_t full[G::STAGES], inboxfull;
    __shared__ float s_max[PT][16];
    const uint32_t sbase = smem_u32(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t rank = cluster_rank(), cs = cluster_size();
    const int req = blockIdx.z, hk = blockIdx.y;
    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&p.kvmap) : "memory");
        for (int s = 0; s < G::STAGES; s++) mbar_init(smem_u32(full + s), 1);
        mbar_init(smem_u32(&inboxfull), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();
    if (cs > 1) cluster_arrive_relaxed();

    const int prefix = p.prefix[req];
    const int nact = min((prefix + p.tail + kKeyBlock - 1) / kKeyBlock, p.nkb);
    const int b0 = nact * (int)rank / (int)cs, b1 = nact * ((int)rank + 1) / (int)cs;       // this CTA's key blocks
    const int new0 = prefix + p.write_off;                              // first cache row this pass writes
    const int krow = p.row0 + req * p.req_rows + hk * p.cap, vrow = krow + p.Hkv * p.cap;
    auto load = [&](int b) {                                            // one thread
        const uint32_t bar = smem_u32(full + (b - b0) % G::STAGES), dst = sbase + ((b - b0) % G::STAGES) * G::BLOCK;
        mbar_expect_tx(bar, G::BLOCK);
#pragma unroll
        for (int x = 0; x < HD / 64; x++) {
            tma_box(dst + x * 8192, &p.kvmap, x * 64, krow + b * kKeyBlock, bar);
            tma_box(dst + (HD / 64 + x) * 8192, &p.kvmap, x * 64, vrow + b * kKeyBlock, bar);
        }
    };
    const int committed = min(b1, new0 / kKeyBlock);                    // blocks below it hold no row of this pass
    const int asked = max(b0, min(committed, b0 + G::STAGES));
    constexpr int kLoader = kAWarps - 1;
    if (warp == kLoader) {
        if (elect_one())
            for (int b = b0; b < asked; b++) load(b);
        __syncwarp();
    }
    const int Gq = p.Hq / p.Hkv, rows = p.mr * Gq;
    const int part = warp, lr = g;                                       // this thread's rows: lr, lr + 8
    const bool v0 = lr < rows, v1 = lr + 8 < rows, busy = b0 < b1;
    const int nslot = (rows + (int)cs - 1) / (int)cs, row_lo = (int)rank * nslot, mine_rows = min(nslot, rows - row_lo);     // rows this CTA finishes
    if (cs > 1 && threadIdx.x == 0)                                     // what will be stored here: (max, sum) from all, outputs from those with keys
        mbar_expect_tx(smem_u32(&inboxfull), max(mine_rows, 0) * ((int)cs * PT * 8 + min(nact, (int)cs) * HD * 4));
    if (cs > 1) cluster_wait();                                         // the peers have started: they may be stored to
    pdl_wait();
    if (warp == kLoader) {
        if (elect_one()) {
            asm volatile("fence.proxy.async;\n" ::: "memory");                 // rows appended by the previous kernel's ordinary stores
            for (int b = asked; b < min(b1, b0 + G::STAGES); b++) load(b);
        }
        __syncwarp();
    }
    // queries -> shared memory, 16 bytes a thread
#pragma unroll 2
    for (int i = threadIdx.x; i < G::ROWS * HD / 8; i += kAWarps * 32) {
        const int r = i / (HD / 8), v = i % (HD / 8);
        uint4 q = make_uint4(0, 0, 0, 0);
        if (r < rows) {
            const int tok = r / Gq;
            q = __ldcg(reinterpret_cast<const uint4*>(p.q + (size_t)(req * p.mr + tok) * p.pitch + (size_t)(hk * Gq + r - tok * Gq) * HD) + v);
        }
        *reinterpret_cast<uint4*>(smem + G::Q + r * HD * 2 + ((v ^ (r & 7)) << 4)) = q;
    }
    const unsigned long long mk0 = v0 ? p.mask[req * p.mr + lr / Gq] : 0ull;
    const unsigned long long mk1 = v1 ? p.mask[req * p.mr + (lr + 8) / Gq] : 0ull;
    __syncthreads();

    constexpr int KT = 8 / PT;                                          // 8-key columns of a warp in the first matmul
    constexpr int ND = HD / PT / 8;                                     // 8-dim columns in the second
    float mrun0 = -INFINITY, mrun1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    float o[ND][4];
#pragma unroll
    for (int nd = 0; nd < ND; nd++) o[nd][0] = o[nd][1] = o[nd][2] = o[nd][3] = 0.f;
    const uint32_t arow = (uint32_t)(lane & 15), avec = (uint32_t)(lane >> 4);                           // fragments of Q and P
    const uint32_t krow_l = (uint32_t)(lane & 7), kvec_l = (uint32_t)(lane >> 3);                        // of K
    const uint32_t vrow_l = (uint32_t)(((lane >> 3) & 1) * 8 + (lane & 7)), vvec_l = (uint32_t)(lane >> 4);    // and of V
    const uint32_t qaddr = sbase + G::Q + arow * (HD * 2), paddr = sbase + G::P;

#pragma unroll 1
    for (int b = b0; b < b1; b++) {
        const int st = (b - b0) % G::STAGES;
        mbar_wait_reported(smem_u32(full + st), ((b - b0) / G::STAGES) & 1, p.polls, p.err, 29);
        __syncwarp();
        if (busy) {
            const uint32_t sk = sbase + st * G::BLOCK, sv = sk + (HD / 64) * 8192;
            if (b == b1 - 1)                                             // rows of V past the last: 0 x Inf or NaN would be NaN
#pragma unroll 1
                for (int k = (prefix + p.tail - b * kKeyBlock) * 8 + (int)threadIdx.x; k < kKeyBlock * 8; k += kAWarps * 32)
#pragma unroll
                    for (int x = 0; x < HD / 64; x++)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(sv + x * 8192 + k * 16), "r"(0) : "memory");
            // scores of this warp's keys
            const int k0 = part * KT * 8;
            float s[KT][4], s1[KT][4];                                   // (even and odd steps apart: chains of half the length)
#pragma unroll
            for (int nt = 0; nt < KT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) s[nt][e] = s1[nt][e] = 0.f;
#pragma unroll 2
            for (int ks = 0; ks < HD / 16; ks += 2) {
                uint32_t qa[4], qb[4];
                ldsm4(qa, qaddr + (((ks * 2 + avec) ^ (arow & 7)) << 4));
                ldsm4(qb, qaddr + (((ks * 2 + 2 + avec) ^ (arow & 7)) << 4));
#pragma unroll
                for (int nt = 0; nt < KT; nt++) {
                    uint32_t kf[4];
                    ldsm4(kf, sk + kv_swz(k0 + nt * 8 + krow_l, ks * 2 + kvec_l));
                    mma_m16n8k16(s[nt], qa[0], qa[1], qa[2], qa[3], kf[0], kf[1]);
                    mma_m16n8k16(s1[nt], qb[0], qb[1], qb[2], qb[3], kf[2], kf[3]);
                }
            }
#pragma unroll
            for (int nt = 0; nt < KT; nt++)
#pragma unroll
                for (int e = 0; e < 4; e++) s[nt][e] += s1[nt][e];
            float mx0 = -INFINITY, mx1 = -INFINITY;
            const int j0 = b * kKeyBlock + k0 + 2 * t - prefix;          // tail row of the thread's first key
            const bool open = b * kKeyBlock + kKeyBlock <= prefix;       // committed rows only
#pragma unroll
            for (int nt = 0; nt < KT; nt++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    bool vis0 = v0, vis1 = v1;
                    const int j = j0 + nt * 8 + e;
                    if (!open && j >= 0) {
                        vis0 = v0 && j < p.tail && ((mk0 >> (j & 63)) & 1ull);
                        vis1 = v1 && j < p.tail && ((mk1 >> (j & 63)) & 1ull);
                    }
                    s[nt][e] = vis0 ? s[nt][e] * p.scale_log2 : -INFINITY;
                    s[nt][2 + e] = vis1 ? s[nt][2 + e] * p.scale_log2 : -INFINITY;
                    mx0 = fmaxf(mx0, s[nt][e]);
                    mx1 = fmaxf(mx1, s[nt][2 + e]);
                }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            if (t == 0) {
                s_max[part][g] = mx0;
                s_max[part][g + 8] = mx1;
            }
            __syncthreads();
            mx0 = mrun0;
            mx1 = mrun1;
#pragma unroll
            for (int i = 0; i < PT; i++) {
                mx0 = fmaxf(mx0, s_max[i][g]);
                mx1 = fmaxf(mx1, s_max[i][g + 8]);
            }
            const float base0 = (mx0 == -INFINITY) ? 0.f : mx0;
            const float base1 = (mx1 == -INFINITY) ? 0.f : mx1;
            const float al0 = (mrun0 == -INFINITY) ? 0.f : exp2f(mrun0 - base0);
            const float al1 = (mrun1 == -INFINITY) ? 0.f : exp2f(mrun1 - base1);
            l0 *= al0; l1 *= al1;
            mrun0 = mx0; mrun1 = mx1;
#pragma unroll
            for (int nt = 0; nt < KT; nt++) {
                const __half2 h0 = __floats2half2_rn(exp2f(s[nt][0] - base0), exp2f(s[nt][1] - base0));
                const __half2 h1 = __floats2half2_rn(exp2f(s[nt][2] - base1), exp2f(s[nt][3] - base1));
                // the sum uses the rounded probabilities so that numerator and denominator agree
                l0 += __low2float(h0) + __high2float(h0);
                l1 += __low2float(h1) + __high2float(h1);
                unsigned char* d = smem + G::P + g * 128 + (((part * KT + nt) ^ g) << 4) + t * 4;      // (rows g and g + 8: the same swizzle)
                *reinterpret_cast<__half2*>(d) = h0;
                *reinterpret_cast<__half2*>(d + 1024) = h1;
            }
#pragma unroll
            for (int nd = 0; nd < ND; nd++) { o[nd][0] *= al0; o[nd][1] *= al0; o[nd][2] *= al1; o[nd][3] *= al1; }
            __syncthreads();
            // this warp's dims of the output, over all keys of the block
#pragma unroll 2
            for (int ks = 0; ks < 4; ks++) {
                uint32_t pa[4];
                ldsm4(pa, paddr + arow * 128 + (((ks * 2 + avec) ^ (arow & 7)) << 4));
#pragma unroll
                for (int nd = 0; nd < ND; nd += 2) {
                    uint32_t vb[4];
                    ldsm4_t(vb, sv + kv_swz(ks * 16 + vrow_l, part * ND + nd + vvec_l));
                    mma_m16n8k16(o[nd], pa[0], pa[1], pa[2], pa[3], vb[0], vb[1]);
                    mma_m16n8k16(o[nd + 1], pa[0], pa[1], pa[2], pa[3], vb[2], vb[3]);
                }
            }
        }
        if (b + G::STAGES < b1) {                                        // the stage is asked for again
            __syncthreads();
            if (warp == kLoader) {
                if (elect_one()) load(b + G::STAGES);
                __syncwarp();
            }
        }
    }
    // ---- partial states -> the CTA that finishes each row
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
#pragma unroll
    for (int hrow = 0; hrow < 2; hrow++) {
        const int row = lr + 8 * hrow;
        if (row < rows) {
            const uint32_t dst = row / nslot, sl = row - dst * nslot;    // (a warp's rows: mostly one CTA)
            const uint32_t ml_at = sbase + G::INBOX_ML + ((rank * PT + part) * nslot + sl) * 8;
            const uint32_t out_at = sbase + G::INBOX + ((rank * nslot + sl) * G::OP + part * ND * 8 + 2 * t) * 4;
            const uint32_t ml[2] = {__float_as_uint(hrow ? mrun1 : mrun0), __float_as_uint(hrow ? l1 : l0)};
            if (cs > 1) {                                                // (a store counts its own bytes at the peer's barrier)
                const uint32_t bar = peer_addr(smem_u32(&inboxfull), dst), at = peer_addr(out_at, dst);
                if (t == 0) st_async<2>(peer_addr(ml_at, dst), ml, bar);
                if (busy) {
#pragma unroll
                    for (int nd = 0; nd < ND; nd++) {
                        const uint32_t x[2] = {__float_as_uint(o[nd][2 * hrow]), __float_as_uint(o[nd][2 * hrow + 1])};
                        st_async<2>(at + nd * 32, x, bar);
                    }
                }
            } else {                                                     // (st.async belongs to clusters)
                if (t == 0) asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(ml_at), "r"(ml[0]), "r"(ml[1]) : "memory");
                if (busy) {
#pragma unroll
                    for (int nd = 0; nd < ND; nd++)
                        asm volatile("st.shared.v2.f32 [%0], {%1, %2};\n" ::"r"(out_at + nd * 32), "f"(o[nd][2 * hrow]), "f"(o[nd][2 * hrow + 1]) : "memory");
                }
            }
        }
    }
    if (cs > 1) {
        inbox_wait(smem_u32(&inboxfull), p.polls, p.err, 25);
        __syncwarp();
    } else {
        __syncthreads();
    }
    // ---- merge: one warp per row, CTAs in key order
#pragma unroll 1
    for (int j = warp; j < mine_rows; j += kAWarps) {
        constexpr int C = HD / 32;
        const float2* ml = reinterpret_cast<const float2*>(smem + G::INBOX_ML) + j;
        const float2 mine = lane < (int)cs * PT ? ml[lane * nslot] : make_float2(-INFINITY, 0.f);     // lane: (source, part); at most 32
        float mstar = mine.x;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) mstar = fmaxf(mstar, __shfl_xor_sync(0xffffffffu, mstar, i));
        const float w = mine.x == -INFINITY ? 0.f : exp2f(mine.x - mstar);
        float den = w * mine.y;
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) den += __shfl_xor_sync(0xffffffffu, den, i);
        float acc[C];
#pragma unroll
        for (int c = 0; c < C; c++) acc[c] = 0.f;
        const float* v = reinterpret_cast<const float*>(smem + G::INBOX) + j * G::OP + lane * C;
#pragma unroll 2
        for (int i = 0; i < (int)cs; i++) {
            const float wi = __shfl_sync(0xffffffffu, w, i * PT);
            if (wi != 0.f) {                                             // (an idle source has left no output)
#pragma unroll
                for (int c = 0; c < C; c++) acc[c] += wi * v[i * nslot * G::OP + c];
            }
        }
        const float inv = den > 0.f ? 1.f / den : 0.f;
        const int gr = row_lo + j, tok = gr / Gq;
        __half* dst = p.out + (size_t)(req * p.mr + tok) * p.Hq * HD + (size_t)(hk * Gq + gr - tok * Gq) * HD + lane * C;
        __align__(8) __half ov[C];
#pragma unroll
        for (int c = 0; c < C; c++) ov[c] = __float2half_rn(acc[c] * inv);
        if (C == 4) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(ov);
        else *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(ov);
    }
}

// ================================================================================ host
// Cluster size along K for `tiles` row tiles of `nch` chunks, by a cost (in chunks) fitted on B200 to passes of four model shapes with 1, 8, 16
// and 32 tokens, one kernel's size changed at a time around the choice: a chunk, one behind the three that are expanded before the wait as
// much again; a source of the reduction 0.38 and 0.007 a token; clusters that nearly fill what runs at once (eight GPCs of at least 16 SMs,
// two CTAs each) start late, and beyond it run as a second wave (36 clusters of 7 or 48 of 6 added 2 to 8 us a kernel): not taken, nor eights
// of more than 28 tiles (32 x 112 chunks: + 0.7 to 1.7 us).  On average 0.02 us a kernel behind the best of the 64 cases.  (The terms fitted
// when an exchange cost 0.5 us more kept to half the cluster: 24 x 16 chunks, 32 tokens - 2.2 us with 8 instead of 4, 128 x 16 - 2.8 with 2
// instead of none.)
int plan_cluster(int tiles, int nch, int tokens) {
    int best = 1;
    double best_cost = 1e30;
    for (int cs = 1; cs <= kMaxCluster && cs <= nch && (cs == 1 || tiles <= 8 * (32 / cs)) && (cs < 8 || tiles <= 28); cs++) {
        const int n = ((nch + cs - 1) / cs) * ((tiles * cs + 295) / 296);
        const double cost = n + std::max(0, n - 3) + (0.38 + 0.007 * tokens) * cs + (cs > 1 ? std::max(0.0, tiles / (8.0 * (32 / cs)) - 0.8) * 8.4 : 0.0);
        if (cost < best_cost - 1e-9) { best_cost = cost; best = cs; }
    }
    return best;
}
// Clusters of 1 .. 8 CTAs that find SMs of their own (148 SMs in GPCs of 16 to 20; cudaOccupancyMaxActiveClusters at one CTA per SM).
constexpr int kOwnSms[kMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};

// The same for a matmul on its own, which has nothing but its like before and behind it: in microseconds but for a constant, fitted to 40
// shapes from 128 x 256 to 8192 x 8192 of 1 to 32 rows with every size; 0.3 % behind the best of each on average, 6 % at most.
// Re-laid-out weights: a chunk 0.2, behind the third 0.05 more, a source of the reduction 0.04, two groups of tokens to finish 0.2; a CTA that
// shares its SM comes up 0.1 to 1.4 later.  (With the terms of exchanges half a microsecond dearer: 32 x 896 x 896 3.7 us in threes, 3.0 in
// sevens; 32 x 512 x 2048 3.7, 3.3 in eights; 8 x 256 x 512 2.8, 2.1 in fours.)
// As quantised nothing is expanded before the wait, and two CTAs of an SM then work at the same time: each takes nearly twice as long (2560 x
// 9728: 9.2 us in sixes, 120 CTAs, 11.8 in sevens, 140 CTAs).  (Before: 8 x 512 x 2048 4.5 in fours, 3.7 in eights; 16 x 896 x 896 4.0 and 3.4.)
int plan_alone(int tiles, int nch, int tokens, int group, bool as_quantised) {
    int best = 1;
    double best_cost = 1e30;
    const int groups = (tokens + group - 1) / group;
    for (int cs = 1; cs <= kMaxCluster && cs <= nch && (cs == 1 || tiles <= 8 * (32 / cs)); cs++) {
        const int n = ((nch + cs - 1) / cs) * ((tiles * cs + 295) / 296), finish = ((groups + cs - 1) / cs + 1) / 2;
        const bool shared = tiles > kOwnSms[cs];
        const double part = std::min(1.0, std::max(0.0, (double)tiles / kOwnSms[cs] - 1));
        const double cost = as_quantised ? n * (shared ? 0.38 : 0.2) + (cs > 1 ? 0.17 : 0) + 0.003 * cs + 0.05 * finish + 0.2 * part
                                         : n * 0.2 + std::max(0, n - 3) * 0.05 + (cs > 1 ? 0.04 * cs : 0) + 0.2 * finish + (shared ? 0.1 : 0) + 1.3 * part;
        if (cost < best_cost - 1e-9) { best_cost = cost; best = cs; }
    }
    return best;
}

template <int NT, int TQ, int KIND, bool TABLE = false, bool WIDE = false, bool FAST = false>
int launch_dense(DenseParams& p, int split, cudaStream_t stream) {
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(dense_kernel<NT, KIND, TQ, TABLE, WIDE, FAST>, DGeo<NT, TQ>::SMEM, done, KIND != D_ROWS)) return check_launch();
    const int nch = p.K / kChunkK;
    const int tiles = KIND == D_SILU ? p.N / 64 : (p.N + kTileRows - 1) / kTileRows, wide = WIDE ? (p.M + NT - 1) / NT : 1;
    const int cs = split > 0 && split <= std::min(kMaxCluster, nch) ? split
                   : KIND == D_PLAIN || KIND == D_ROWS                ? plan_alone(tiles, nch, p.M, TQ, KIND == D_ROWS)
                                                                      : plan_cluster(tiles * wide, nch, std::min(p.M, NT));
    constexpr int cap = 296;
    auto launch = [&](int lo, int n, int cluster) {
        p.tile_lo = lo;
        p.tiles = lo + n;
        return launch_chain(dense_kernel<NT, KIND, TQ, TABLE, WIDE, FAST>, dim3(cluster > 1 ? n * cluster : std::min(n, cap), wide), kDThreads, DGeo<NT, TQ>::SMEM, cluster, stream, p);
    };
    // Whole waves of tiles, then what is left over as a launch of its own with K split over clusters: alone it would take as long
    // as a whole wave.
    const int rest = cs == 1 && tiles > cap ? tiles % cap : 0, rest_cs = rest > 0 ? std::min({cap / rest, kMaxCluster, nch}) : 1;
    if (WIDE || rest_cs < 2) return launch(0, tiles, cs);
    const int rc = launch(0, tiles - rest, 1);
    return rc != B200_OK ? rc : launch(tiles - rest, rest, rest_cs);
}

// Clusters of as many key ranges as still run at once, two CTAs to an SM.  `split` as b200_forward_desc.attn_split_blocks.
template <int HD>
int launch_attention(DAttn& a, int nreq, int split, cudaStream_t stream) {
    using G = DAGeo<HD>;
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(attention_kernel<HD>, G::SMEM, done, true)) return check_launch();
    const int clusters = a.Hkv * nreq;
    int cs = std::min(a.nkb, kMaxCluster);
    while (split >= 0 && cs > 1 && clusters > 8 * (32 / cs)) cs--;
    if (split > 0 && a.nkb < split) cs = 1;
    return launch_chain(attention_kernel<HD>, dim3(cs, a.Hkv, nreq), kAWarps * 32, G::SMEM, cs, stream, a);
}

// TABLE: the kernels take a layer's pointers from the table in device memory, in stream order like everything else.  (Variants of
// their own: the load is ahead of a CTA's first weights.)
template <int NT, int TQ, bool TABLE, bool FAST>
int run_chain(const ChainArgs& c, cudaStream_t st) {
    const b200_forward_desc* d = c.d;
    const int M = d->M, H = d->hidden, I = d->intermediate, hd = d->head_dim, nreq = d->requests > 1 ? d->requests : 1;
    const int nq = d->n_heads * hd, nqkv = (d->n_heads + 2 * d->n_kv_heads) * hd;
    auto on = [&](int kind) { return d->phase_mask == 0 || ((d->phase_mask >> kind) & 1); };
    CUtensorMap hw_map, attn_map, act_map;
    auto xmap = [&](CUtensorMap* m, const void* x, int width) {
        return make_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, width, M, (uint64_t)width * 2, 64, NT, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    };
    int rc;
    if ((rc = xmap(&hw_map, d->hw, H)) || (rc = xmap(&attn_map, d->attn, nq)) || (rc = xmap(&act_map, d->act, I))) return rc;

    DenseParams p{};
    p.ssq = c.ssq; p.H = H; p.eps = d->rms_eps; p.M = M; p.err = c.err; p.polls = wait_polls(kWaitPolls, kFirmPolls / 2);
    p.h = static_cast<__half*>(d->h); p.hw = static_cast<__half*>(d->hw);
    p.cs = c.cs; p.prefix = d->prefix; p.Hq = d->n_heads; p.Hkv = d->n_kv_heads; p.hd = hd; p.cap = d->cache_rows;
    p.write_off = d->write_off; p.mr = M / nreq;
    const size_t half_stride = (size_t)d->n_kv_heads * d->cache_rows * hd;
    p.req_stride = (size_t)d->n_layers * 2 * half_stride;
    p.row_index = d->row_index; p.rows_out = d->rows_out;
    FlashArgs a{};
    a.q = d->qkv; a.kv = d->kv_cache; a.kv_rows = (uint64_t)nreq * d->n_layers * 2 * d->n_kv_heads * d->cache_rows;
    a.out = d->attn; a.tokens = M; a.Hq = d->n_heads; a.Hkv = d->n_kv_heads; a.hd = hd; a.cap = d->cache_rows;
    a.scale_log2 = d->attn_scale * kLog2e; a.err = c.err; a.polls = p.polls;
    a.mask = d->mask; a.prefix = d->prefix; a.nreq = nreq; a.mr = p.mr; a.tail = d->tail; a.write_off = d->write_off;
    a.nkb = (d->cache_rows + 63) / 64; a.split = d->attn_split_blocks; a.req_rows = d->n_layers * 2 * d->n_kv_heads * d->cache_rows;
    FlashPlan flash{};
    if ((rc = flash_decode_plan(a, &flash)) != B200_OK) return rc;
    DAttn one{};
    one.kvmap = flash.kvmap; one.q = static_cast<const __half*>(d->qkv); one.pitch = nqkv; one.mask = d->mask; one.prefix = d->prefix;
    one.out = static_cast<__half*>(d->attn); one.Hq = d->n_heads; one.Hkv = d->n_kv_heads; one.mr = p.mr; one.tail = d->tail; one.nkb = a.nkb;
    one.req_rows = a.req_rows; one.cap = d->cache_rows; one.write_off = d->write_off; one.scale_log2 = a.scale_log2; one.err = c.err; one.polls = p.polls;
    // Up to 16 query rows of a kv head (a token or two) mma.sync has the shorter chain: next token of the 0.5B shape 455 against 470 us, there 568
    // against 583 with 3000 cached.  At head dim 128 the tensor memory's wins on many cached rows (8 layers of the 7B shape behind 100, 900, 3000,
    // 12000 of them: mma.sync 423, 432, 465, 617 us, the other 425, 430, 453, 559); how many there are only the device knows, so the cache's
    // capacity decides, and few rows in a large cache take up to 1 % longer.  Beyond 16 rows: 0.5B, 8 tokens, 300 cached 493 against 495, 3000 cached
    // 605 against 666.
    const bool few = p.mr * (d->n_heads / d->n_kv_heads) <= DAGeo<64>::ROWS && (hd == 64 || a.nkb <= 16);

    const void* const* layers = TABLE ? static_cast<const void* const*>(d->layer_table) : c.layers;      // (not read here with TABLE)
    auto given = [&](const void* const* L, int i) { return TABLE ? nullptr : L[i]; };
    if (on(0) || TABLE) {                                       // (what makes the table safe to read ahead of a kernel's wait)
        launch_kernel(embed_kernel, dim3(M), dim3(256), 0, st, d->tokens, d->pos, d->embed_wq, static_cast<const __half*>(d->embed_scales),
                      static_cast<const __half*>(d->embed_biases), static_cast<const __half*>(given(layers, 6)), p.h, p.hw, p.ssq, c.cs, d->inv_freq,
                      d->rope_scaling, H, d->vocab, hd / 2, TABLE ? layers + 6 : nullptr);
        if ((rc = check_launch()) != B200_OK) return rc;
    }
    for (int l = 0; l < d->n_layers; l++) {
        const void* const* L = layers + (size_t)l * 8;       // qkv, qkv bias, o, gate, up, down, input norm, post norm
        auto weights = [&](int i, int n) {
            for (int j = 0; j < n; j++) p.w[j] = static_cast<const unsigned char*>(given(L, i + j));
            p.tw = L + i;
        };
        if (on(1)) {
            p.xmap = hw_map; weights(0, 1); p.bias = static_cast<const __half*>(given(L, 1)); p.tv = L + 1; p.y = static_cast<__half*>(d->qkv);
            p.N = nqkv; p.K = H;
            p.kc = static_cast<__half*>(d->kv_cache) + (size_t)l * 2 * half_stride;
            p.vc = p.kc + half_stride;
            if ((rc = launch_dense<NT, TQ, D_QKV, TABLE, false, FAST>(p, c.splits[0], st)) != B200_OK) return rc;
        }
        if (on(2)) {
            const int row0 = l * 2 * d->n_kv_heads * d->cache_rows;
            one.row0 = row0;
            if (few) rc = hd == 128 ? launch_attention<128>(one, nreq, d->attn_split_blocks, st) : launch_attention<64>(one, nreq, d->attn_split_blocks, st);
            else rc = flash_decode(a, flash, row0, st);
            if (rc != B200_OK) return rc;
        }
        p.bias = nullptr;
        if (on(4)) {
            p.xmap = attn_map; weights(2, 1); p.wn = static_cast<const __half*>(given(L, 7)); p.tv = L + 7; p.N = H; p.K = nq;
            if ((rc = launch_dense<NT, TQ, D_RESID, TABLE, false, FAST>(p, c.splits[1], st)) != B200_OK) return rc;
        }
        if (on(5)) {
            p.xmap = hw_map; weights(3, 2); p.y = static_cast<__half*>(d->act); p.N = I; p.K = H;
            if ((rc = launch_dense<NT, TQ, D_SILU, TABLE, false, FAST>(p, c.splits[2], st)) != B200_OK) return rc;
        }
        if (on(6)) {
            const bool more = l + 1 < d->n_layers;
            p.xmap = act_map; weights(5, 1); p.wn = static_cast<const __half*>(more ? given(L, 8 + 6) : d->final_norm); p.tv = more ? L + 8 + 6 : nullptr;
            p.N = H; p.K = I;
            if ((rc = launch_dense<NT, TQ, D_RESID, TABLE, false, FAST>(p, c.splits[3], st)) != B200_OK) return rc;
        }
    }
    if (on(7)) {
        p.xmap = hw_map; p.w[0] = static_cast<const unsigned char*>(d->lm_head_tiled); p.y = static_cast<__half*>(d->logits);
        p.N = d->head_rows > 0 ? d->head_rows : d->vocab; p.K = H;
        if ((rc = launch_dense<NT, TQ, D_HEAD, false, false, FAST>(p, c.splits[4], st)) != B200_OK) return rc;
    }
    return B200_OK;
}

// The layers of a prompt pass: as run_chain, in tiles of 32 tokens side by side, with the norms as kernels between them.
int run_prompt(const ChainPrompt& c, cudaStream_t st) {
    const b200_prefill_desc* d = c.d;
    const int n = d->n, H = d->hidden, I = d->intermediate, hd = d->head_dim, nq = d->n_heads * hd, nqkv = (d->n_heads + 2 * d->n_kv_heads) * hd;
    CUtensorMap xn_map, attn_map, act_map;
    auto xmap = [&](CUtensorMap* m, const void* x, int width) {
        return make_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, width, n, (uint64_t)width * 2, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    };
    int rc;
    if ((rc = xmap(&xn_map, d->xn, H)) || (rc = xmap(&attn_map, d->attn, nq)) || (rc = xmap(&act_map, d->act, I))) return rc;
    DenseParams p{};
    p.M = p.mr = n; p.err = c.err; p.polls = wait_polls(kWaitPolls, kFirmPolls / 2);
    p.h = static_cast<__half*>(d->h);
    p.cs = c.cs; p.write_off = d->off; p.Hq = d->n_heads; p.Hkv = d->n_kv_heads; p.hd = hd; p.cap = d->cache_rows;
    const size_t half = (size_t)d->n_kv_heads * d->cache_rows * hd;
    for (int l = 0; l < d->n_layers; l++) {
        const void* const* L = d->layers + (size_t)l * 8;       // qkv, qkv bias, o, gate, up, down, input norm, post norm
        auto weights = [&](int i, int count) {
            for (int j = 0; j < count; j++) p.w[j] = static_cast<const unsigned char*>(L[i + j]);
        };
        if ((rc = c.norm(c.context, L[6], l == 0, st)) != B200_OK) return rc;
        p.xmap = xn_map; weights(0, 1); p.bias = static_cast<const __half*>(L[1]); p.y = static_cast<__half*>(d->qkv); p.N = nqkv; p.K = H;
        p.kc = static_cast<__half*>(d->kv_cache) + (size_t)l * 2 * half;
        p.vc = p.kc + half;
        if ((rc = launch_dense<32, 4, D_QKV, false, true>(p, 0, st)) != B200_OK) return rc;
        if ((rc = c.attention(c.context, l * 2 * d->n_kv_heads * d->cache_rows, st)) != B200_OK) return rc;
        p.bias = nullptr;
        p.xmap = attn_map; weights(2, 1); p.N = H; p.K = nq;
        if ((rc = launch_dense<32, 4, D_RESID, false, true>(p, 0, st)) != B200_OK) return rc;
        if ((rc = c.norm(c.context, L[7], false, st)) != B200_OK) return rc;
        p.xmap = xn_map; weights(3, 2); p.y = static_cast<__half*>(d->act); p.N = I; p.K = H;
        if ((rc = launch_dense<32, 4, D_SILU, false, true>(p, 0, st)) != B200_OK) return rc;
        p.xmap = act_map; weights(5, 1); p.N = H; p.K = I;
        if ((rc = launch_dense<32, 4, D_RESID, false, true>(p, 0, st)) != B200_OK) return rc;
    }
    return B200_OK;
}

template <int NT, int TQ>
int run_matmul(const ChainMatmul& c, cudaStream_t st) {
    DenseParams p{};
    int rc = make_map_2d(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, c.x, c.K, c.M, (uint64_t)c.K * 2, 64, NT, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (rc != B200_OK) return rc;
    p.bias = static_cast<const __half*>(c.bias);
    p.y = static_cast<__half*>(c.y);
    p.M = p.mr = c.M; p.N = c.N; p.K = c.K; p.hd = 64; p.err = c.err; p.polls = wait_polls(kWaitPolls, kFirmPolls / 2);
    if (c.scales == nullptr) {
        p.w[0] = static_cast<const unsigned char*>(c.w);
        return launch_dense<NT, TQ, D_PLAIN>(p, 0, st);
    }
    p.sc = static_cast<const __half*>(c.scales);
    p.bi = static_cast<const __half*>(c.biases);
    rc = make_map_2d(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, c.w, c.K / 2, c.N, c.K / 2, 64, kTileRows, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    return rc != B200_OK ? rc : launch_dense<NT, TQ, D_ROWS>(p, 0, st);
}

}  // namespace

// Against the large-M kernel, over the shapes above, us here / there.  The clusters add up K without going through memory and the CTAs are
// half as large, which counts for more the fewer chunks an SM has; its four groups of dequant warps against three win with many.
// Re-laid-out: up to 2047 chunks (32 rows: 896 x 896 3.0 / 3.9, 4096 x 4096 6.5 / 8.4, 5120 x 5120 7.8 / 9.4, 32000 x 1024 8.7 / 9.3; 16384 x
// 2048 7.7 to 8.8 / 7.8 to 8.3), and where it has to split K, which it does through memory, up to 4096 (32 x 4096 x 8192 9.2 / 10.8, 32 x 8192
// x 8192 13.6 / 17.6; 18944 x 3584 12.4 to 14.4 / 11.9 to 12.5, 3584 x 18944 the same).
// As quantised, where weights have to wait, scales are to be fetched and pairs reordered: always up to 320 chunks (32 rows: 896 x 896 3.7 /
// 4.8, 512 x 2048 4.2 / 6.3; the smallest only up to 16 rows, 128 x 256 2.7 / 2.9, 32 rows 3.4 / 3.0), up to 1024 if no SM has two CTAs of
// it (32 x 4608 x 3584 8.8 / 9.2), up to 2048 if moreover K is split and most SMs have one (8 x 4096 x 8192 10.6 / 11.7, 5120 x 5120 9.5 /
// 10.5; 6144 x 4096 with 96 CTAs the same, 16384 x 2048 10.3 / 9.2, 6144 x 6144 12.1 / 11.5).
bool chain_matmul_wins(int M, int N, int K, bool as_quantised) {
    if (M > 32) return false;
    const int tiles = (N + kTileRows - 1) / kTileRows, nch = K / kChunkK;
    const long long chunks = (long long)tiles * nch;
    if (!as_quantised) return chunks < 2048 || (tiles <= 64 && chunks <= 4096);
    if (chunks < (M <= 16 ? 1 : 8) || chunks > 2048) return false;
    const int cs = plan_alone(tiles, nch, M, M <= 8 ? 2 : 4, true);
    return chunks <= 320 || (tiles <= kOwnSms[cs] && (chunks <= 1024 || (cs > 1 && tiles * cs >= 108)));
}

int chain_matmul(const ChainMatmul& c, cudaStream_t st) {
    return c.M <= 8 ? run_matmul<16, 2>(c, st) : (c.M <= 16 ? run_matmul<16, 4>(c, st) : run_matmul<32, 4>(c, st));
}

template <bool TABLE, bool FAST>
static int forward_chain_rows(const ChainArgs& a, cudaStream_t stream) {
    return a.d->M <= 8 ? run_chain<16, 2, TABLE, FAST>(a, stream) : (a.d->M <= 16 ? run_chain<16, 4, TABLE, FAST>(a, stream) : run_chain<32, 4, TABLE, FAST>(a, stream));
}

int chain_prompt(const ChainPrompt& c, cudaStream_t st) { return run_prompt(c, st); }

int forward_chain(const ChainArgs& a, cudaStream_t stream) {
    if (a.layers == nullptr) return forward_chain_rows<true, false>(a, stream);
    return a.d->scales_in_fast_range ? forward_chain_rows<false, true>(a, stream) : forward_chain_rows<false, false>(a, stream);
}

}  // namespace b200
