// Tree-masked and causal attention on the fifth-generation tensor cores, GQA.
//
// CTA = (64 query rows of one kv head, 128 in a prompt pass; key range); a query row is (token, head of the group), so a block of keys is read once for
// the whole group.  Per 64 keys: S = Q K^T (tcgen05, both operands from shared memory as TMA brought them), four threads a row (two in a prompt
// pass) turn its 64 scores in tensor memory into probabilities in place (fp16, two to a column), O += P V (P from tensor memory, V as it lies: keys
// by dims).  Scores are double-buffered, so the tensor cores work on the next block's while a block's softmax runs.
// O is rescaled in tensor memory whenever a row's maximum grows, by the row's threads, once their probabilities of the block are written
// and the block before has been added.  (A maximum kept until exceeded by 2^8 was 1 to 4 % of a pass faster, but the largest weight is
// then rounded, too: 2.9e-4 against 2.2e-4 of relative error, 32 tokens of the 8B shape over 3500 rows.)
// Probabilities are rounded to fp16 and summed as rounded, scores, sums and O are fp32: the rounding points of the mma.sync kernels this
// replaces (32 tokens of the 8B shape over 3500 rows: 20 us a layer there; a causal pass of 1024: 63 us).
//
// A row's threads sit in the same lane of warps 4 apart, which see the same part of tensor memory.  (With one thread a row a block of
// 128 rows took 1540 cycles.)
//
// Decode: the CTAs of a cluster take neighbouring key ranges; each finishes its share of the rows, whose partial outputs the
// others copy into its shared memory (bulk copies between the CTAs, counted by its barrier; as 16-byte stores they took 3.6 us), merged in range order.  Committed blocks are asked for before the wait for the
// kernel that appends this pass's rows.  Prompt passes: a CTA goes through all its keys, or, where few tokens look at a long cache,
// through a range whose partial state a second kernel merges.
// Every wait is bounded; one that runs out sets the error word and goes on.  No copy uses cluster multicast.
#include <algorithm>
#include <atomic>

#include "flash.cuh"
#include "pipeline.cuh"
#include "tensor_map.cuh"
#include "umma.cuh"

namespace b200 {
namespace {

constexpr int kKeyBlock = 64;
constexpr int kTmem = 256;                       // O (HD columns), then two blocks of scores

template <int HD, bool DECODE>
struct FGeo {
    static constexpr int ROWS = DECODE ? 64 : 128;
    static constexpr int PARTS = DECODE ? 4 : 2, KEYS = kKeyBlock / PARTS;       // threads of a row, and keys of each
    // Row warps: 32 rows each by warp % 4, a part by warp / 4.  64 rows leave every other two warps without, of which one copies and one issues MMAs.
    static constexpr int LOADER = DECODE ? 2 : 8, ISSUER = DECODE ? 3 : 9, THREADS = (DECODE ? 14 : 10) * 32;
    static constexpr int QBOX = ROWS * 128;                              // 64 dims of the queries
    static constexpr int KV0 = QBOX * (HD / 64);
    static constexpr int HALF = kKeyBlock * HD * 2;                      // K or V of a block
    static constexpr int STAGES = DECODE && HD == 64 ? 4 : 2;
    static constexpr int END = KV0 + STAGES * 2 * HALF;
    // Once the cluster's MMAs are over: partial outputs of this CTA's rows at the end [row][OP], and those of its share of the rows from all
    // CTAs at the beginning [source][row][OP] (64 rows and a few more).
    static constexpr int OP = HD + 4;                                    // floats: the dims, (max, sum); rows 16 bytes apart in the banks
    static constexpr int OUT = END - ROWS * OP * 4;
    // CTAs of a cluster wait for one another, so none may have to wait for tensor memory behind two of them: no more than two to an SM, and none
    // beside a CTA that takes all of it (csrc/qmm_pair.cu).
    static constexpr int SMEM = std::max(END + 1024, DECODE ? 77 * 1024 : 0);
    static_assert(KV0 % 1024 == 0 && 2 * (SMEM + 4096) <= 227 * 1024 && (!DECODE || (ROWS + 7) * OP * 4 <= OUT), "does not fit");
};

struct FParams {
    CUtensorMap qmap, kvmap;
    __half* out;
    const unsigned long long* mask;
    const int* prefix;
    float* part_o;
    float* part_ml;
    int Hq, Hkv, G, heads, T, hsets, cap, row0;
    int mr, tail, write_off, nkb, req_rows;      // decode
    int n, off, splits;                          // prompt
    float scale_log2;
    int* err;
    int polls;
};

// N-major shared-memory matrix (V: keys by dims), 128-byte swizzle: 64 dims a row of 128 bytes, groups of 8 keys 1024 bytes apart, the next
// 64 dims `box` bytes on.
__device__ __forceinline__ uint64_t sw128_desc_n_major(uint32_t saddr, uint32_t box) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)(box >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
__device__ __forceinline__ void tma_box3(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// Shared memory of this CTA -> that of a CTA of the cluster, counted at a barrier there.
__device__ __forceinline__ void bulk_copy_s2s(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

template <int HD, bool DECODE>
__global__ void __launch_bounds__(FGeo<HD, DECODE>::THREADS) flash_kernel(const __grid_constant__ FParams p) {
    using G = FGeo<HD, DECODE>;
    constexpr int ST = G::STAGES, PT = G::PARTS, KEYS = G::KEYS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    __shared__ uint64_t qfull, kfull[ST], kfree[ST], vfull[ST], vfree[ST], sfull[2], pready[2], pvdone, ofull, inboxfull;
    __shared__ uint32_t s_tmem;
    __shared__ float s_part[2][PT][G::ROWS];                             // what a row's threads tell one another, two blocks in turn
    const uint32_t sbase = smem_u32(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t rank = DECODE ? cluster_rank() : 0, cs = DECODE ? cluster_size() : 1;

    // ---- which rows, which keys
    const int set = DECODE ? (int)blockIdx.y : (int)gridDim.x - 1 - (int)blockIdx.x;      // (prompt: the longest key ranges first)
    const int sets_of_head = DECODE ? (int)gridDim.y / p.Hkv : (int)gridDim.x;
    const int hk = DECODE ? set / sets_of_head : (int)blockIdx.y, in = DECODE ? set - hk * sets_of_head : set;
    const int ts = in / p.hsets, hs = in - ts * p.hsets;                 // token set, head set
    const int req = DECODE ? blockIdx.z : 0, ntok = DECODE ? p.mr : p.n;
    const int tok_base = req * ntok + ts * p.T, toks = min(p.T, ntok - ts * p.T), rows = toks * p.heads;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&p.kvmap) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(&p.qmap) : "memory");
        mbar_init(smem_u32(&qfull), 1);
        for (int s = 0; s < ST; s++) {
            mbar_init(smem_u32(kfull + s), 1);
            mbar_init(smem_u32(kfree + s), 1);
            mbar_init(smem_u32(vfull + s), 1);
            mbar_init(smem_u32(vfree + s), 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(smem_u32(sfull + s), 1);
            mbar_init(smem_u32(pready + s), PT * ((rows + 31) / 32));
        }
        mbar_init(smem_u32(&pvdone), 1);
        mbar_init(smem_u32(&ofull), 1);
        mbar_init(smem_u32(&inboxfull), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == G::ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)), "n"(kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();
    if (DECODE && cs > 1) cluster_arrive_relaxed();

    // Mask and committed length are read ahead of the wait for the kernel before this one: where they are given as memory, that was written
    // before the pass, and what wrote it is complete before any kernel of the pass starts.  A causal pass has them by value (`off`).
    const int prefix = DECODE && p.prefix != nullptr ? p.prefix[req] : p.off;
    int b0, b1;                                                          // this CTA's key blocks
    if (DECODE) {
        const int nact = min((prefix + p.tail + kKeyBlock - 1) / kKeyBlock, p.nkb);
        b0 = nact * (int)rank / (int)cs;
        b1 = nact * ((int)rank + 1) / (int)cs;
    } else {
        const int all = (p.off + ts * p.T + toks - 1) / kKeyBlock + 1, per = (all + p.splits - 1) / p.splits;
        b0 = (int)blockIdx.z * per;
        b1 = min(b0 + per, all);
    }
    const int nb = max(b1 - b0, 0), end = DECODE ? prefix + p.tail : p.off + p.n;      // (first cache row that is nobody's)
    const int nslot = (rows + (int)cs - 1) / (int)cs, row_lo = (int)rank * nslot, mine_rows = min(nslot, rows - row_lo);    // rows this CTA finishes
    if (DECODE && cs > 1 && threadIdx.x == 0)                            // what the cluster will copy here
        mbar_expect_tx(smem_u32(&inboxfull), max(mine_rows, 0) * (int)cs * G::OP * 4);
    const uint32_t tS = tmem + HD;                                       // scores, then probabilities, of block i: + 64 (i & 1)

    if (warp == G::LOADER) {
        // ------------------------------------------------------------------ copies
        const int krow = p.row0 + (DECODE ? req * p.req_rows : 0) + hk * p.cap, vrow = krow + p.Hkv * p.cap;
        // K and V in rings of their own: a block's K is needed one block earlier than its V and is free again as much earlier.  (Behind one
        // barrier the next K came 0.3 us a block late.)
        auto load = [&](int i, int v) {                                  // (one thread)
            const uint32_t bar = smem_u32((v ? vfull : kfull) + i % ST), dst = sbase + G::KV0 + (i % ST) * 2 * G::HALF + v * G::HALF;
            mbar_expect_tx(bar, G::HALF);
#pragma unroll
            for (int x = 0; x < HD / 64; x++) tma_box(dst + x * 8192, &p.kvmap, x * 64, (v ? vrow : krow) + (b0 + i) * kKeyBlock, bar);
        };
        // blocks that hold no row of this pass do not depend on the kernel before this one
        const int early = DECODE ? max(0, min(min(b1, (prefix + p.write_off) / kKeyBlock) - b0, ST)) : 0, first = min(nb, ST);
        if (elect_one())
#pragma unroll 1
            for (int i = 0; i < 2 * early; i++) load(i >> 1, i & 1);
        __syncwarp();
        if (DECODE && cs > 1) cluster_wait();                            // (the peers have started)
        pdl_wait();
        if (elect_one()) {
            // The previous kernel appended rows by ordinary stores.  (On a long cache they are asked for further down only.)
            asm volatile("fence.proxy.async;\n" ::: "memory");
#pragma unroll 1
            for (int i = 2 * early; i < 2 * first; i++) load(i >> 1, i & 1);
        }
        __syncwarp();
#pragma unroll 1
        for (int i = ST; i <= nb; i++) {                                 // K of block i, V of the one before
            if (i < nb) {
                mbar_wait_reported(smem_u32(kfree + i % ST), (i / ST - 1) & 1, p.polls, p.err, 29);
                __syncwarp();
                if (elect_one()) load(i, 0);
                __syncwarp();
            }
            if (i > ST) {
                mbar_wait_reported(smem_u32(vfree + (i - 1) % ST), ((i - 1) / ST - 1) & 1, p.polls, p.err, 29);
                __syncwarp();
                if (elect_one()) load(i - 1, 1);
                __syncwarp();
            }
        }
    } else if (warp == G::ISSUER) {
        // ------------------------------------------------------------------ MMAs
        constexpr uint32_t base = (1u << 4) | ((uint32_t)(128 >> 4) << 24);
        constexpr uint32_t idesc_s = base | ((uint32_t)(kKeyBlock >> 3) << 17), idesc_o = base | (1u << 16) | ((uint32_t)(HD >> 3) << 17);
        const uint64_t qdesc = sw128_desc(sbase), kdesc = sw128_desc(sbase + G::KV0), vdesc = sw128_desc_n_major(sbase + G::KV0 + G::HALF, 8192);
        auto scores = [&](int i) {
            mbar_wait_reported(smem_u32(kfull + i % ST), (i / ST) & 1, p.polls, p.err, 29);
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (elect_one()) {
                const uint32_t d = tS + 64 * (i & 1);
                const uint64_t k0 = kdesc + (i % ST) * (2 * G::HALF / 16);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ks++)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
                                 "l"(qdesc + (ks >> 2) * (G::QBOX / 16) + (ks & 3) * 2), "l"(k0 + (ks >> 2) * (8192 / 16) + (ks & 3) * 2), "r"(idesc_s), "r"(ks)
                                 : "memory");
                commit_to(smem_u32(sfull + (i & 1)));
                commit_to(smem_u32(kfree + i % ST));
            }
            __syncwarp();
        };
        if (DECODE && cs > 1) cluster_wait();
        pdl_wait();
        if (nb > 0) {
            // (the queries, too: the warp that copies has the last blocks to ask for)
            if (elect_one()) {
                asm volatile("fence.proxy.async;\n" ::: "memory");              // (ordinary stores of the previous kernel)
                mbar_expect_tx(smem_u32(&qfull), p.T * p.heads * HD * 2);
#pragma unroll
                for (int x = 0; x < HD / 64; x++) tma_box3(sbase + x * G::QBOX, &p.qmap, x * 64, hk * p.G + hs * p.heads, tok_base, smem_u32(&qfull));
            }
            __syncwarp();
            mbar_wait_reported(smem_u32(&qfull), 0, p.polls, p.err, 28);
            scores(0);
#pragma unroll 1
            for (int i = 0; i < nb; i++) {
                if (i + 1 < nb) {
                    if (i > 0) mbar_wait_reported(smem_u32(&pvdone), (i - 1) & 1, p.polls, p.err, 28);      // (its probabilities stand where the scores go)
                    scores(i + 1);
                }
                mbar_wait_reported(smem_u32(vfull + i % ST), (i / ST) & 1, p.polls, p.err, 29);
                if (i == nb - 1 && end < (b0 + nb) * kKeyBlock) {        // (while the block's softmax runs)
                    // The box reaches past the last row: there is what the cache, or the next head's, holds there.  Its probabilities are 0, and
                    // 0 x Inf or NaN would be NaN in every row.
                    const uint32_t v = sbase + G::KV0 + (i % ST) * 2 * G::HALF + G::HALF;
#pragma unroll 1
                    for (int k = (end - (b0 + i) * kKeyBlock) * 8 + lane; k < kKeyBlock * 8; k += 32)
#pragma unroll
                        for (int x = 0; x < HD / 64; x++)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(v + x * 8192 + k * 16), "r"(0) : "memory");
                    fence_proxy_async();
                    __syncwarp();
                }
                mbar_wait_reported(smem_u32(pready + (i & 1)), (i >> 1) & 1, p.polls, p.err, 28);
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (elect_one()) {
                    const uint64_t v0 = vdesc + (i % ST) * (2 * G::HALF / 16);
                    const uint32_t a0 = tS + 64 * (i & 1);
#pragma unroll
                    for (int ks = 0; ks < kKeyBlock / 16; ks++)
                        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem),
                                     "r"(a0 + ks * 8), "l"(v0 + ks * (2048 / 16)), "r"(idesc_o), "r"(i + ks) : "memory");
                    commit_to(smem_u32(vfree + i % ST));
                    commit_to(smem_u32(&pvdone));
                    if (i == nb - 1) commit_to(smem_u32(&ofull));
                }
                __syncwarp();
            }
        }
    } else if ((warp & 3) * 32 < rows) {
        // ------------------------------------------------------------------ a query row, KEYS keys of a block
        const int part = warp >> 2, r = (warp & 3) * 32 + lane, t = r / p.heads, g = hs * p.heads + r - t * p.heads;
        const bool valid = r < rows && g < p.G;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        auto row_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + (warp & 3)), "n"(PT * 32) : "memory"); };      // the warps of these rows
        if (DECODE && cs > 1) cluster_wait();
        unsigned long long mk = 0;                                       // the tail rows this row sees
        if (DECODE && valid) {
            mk = p.mask != nullptr ? p.mask[tok_base + t] : (2ull << (ts * p.T + t)) - 1;
            if (p.tail < 64) mk &= (1ull << p.tail) - 1;
        }
        const int lim = p.off + ts * p.T + t;                            // prompt: the last key this row sees
        float m = -INFINITY, l = 0.f;
#pragma unroll 1
        for (int i = 0; i < nb; i++) {
            const uint32_t s0 = tS + 64 * (i & 1) + lanes;
            const int key0 = (b0 + i) * kKeyBlock;
            bool all;                                                    // every key of the block is visible to every row of the warp
            unsigned long long vis = ~0ull;
            if (DECODE) {
                const int base = key0 - prefix;                          // tail row of the block's first key
                all = base <= -kKeyBlock;
                if (!all) vis = base >= 0 ? (base < 64 ? mk >> base : 0ull) : (mk << -base) | ((1ull << -base) - 1);
            } else {
                const int c = lim + 1 - key0;
                all = __all_sync(0xffffffffu, c >= kKeyBlock);
                vis = c >= kKeyBlock ? ~0ull : (c <= 0 ? 0ull : (1ull << c) - 1);
            }
            const uint32_t seen = (uint32_t)(vis >> (KEYS * part));
            mbar_wait_reported(smem_u32(sfull + (i & 1)), (i >> 1) & 1, p.polls, p.err, 27);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t raw[KEYS];
            tmem_ld<KEYS>(raw, s0 + KEYS * part);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            float a[KEYS];
#pragma unroll
            for (int j = 0; j < KEYS; j++) a[j] = __uint_as_float(raw[j]) * p.scale_log2;
            if (!all) {
#pragma unroll
                for (int j = 0; j < KEYS; j++)
                    if (!((seen >> j) & 1)) a[j] = -INFINITY;
            }
            float x[4] = {a[0], a[1], a[2], a[3]};
#pragma unroll
            for (int j = 4; j < KEYS; j++) x[j & 3] = fmaxf(x[j & 3], a[j]);
            s_part[i & 1][part][r] = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
            row_sync();                                                  // (all have read their scores, too: the probabilities take the place of the first)
            float mx = s_part[i & 1][0][r];
#pragma unroll
            for (int j = 1; j < PT; j++) mx = fmaxf(mx, s_part[i & 1][j][r]);
            const bool grown = mx > m && r < rows;                       // (rows past the last hold nothing)
            const float al = !grown ? 1.f : (m == -INFINITY ? 0.f : exp2_approx(m - mx));
            if (grown) m = mx;
            const bool rescale = __any_sync(0xffffffffu, grown) && i > 0;       // (the same in all the rows' warps)
            const float ref = m == -INFINITY ? 0.f : m;
            float sum[2] = {0.f, 0.f};
#pragma unroll
            for (int c = 0; c < KEYS; c += 16) {
                uint32_t pk[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const __half2 h = __floats2half2_rn(exp2_approx(a[c + 2 * j] - ref), exp2_approx(a[c + 2 * j + 1] - ref));
                    // the sum uses the rounded probabilities so that numerator and denominator agree
                    sum[0] += __low2float(h);
                    sum[1] += __high2float(h);
                    pk[j] = h2_as_u32(h);
                }
                tmem_st8(s0 + (KEYS * part + c) / 2, pk);
            }
            l = l * al + (sum[0] + sum[1]);
            if (rescale) {
                mbar_wait_reported(smem_u32(&pvdone), (i - 1) & 1, p.polls, p.err, 27);
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
                for (int c = 0; c < HD / PT; c += 16) {
                    uint32_t o[16];
                    tmem_ld<16>(o, tmem + lanes + part * (HD / PT) + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * al);
                    tmem_st8(tmem + lanes + part * (HD / PT) + c, o);
                    tmem_st8(tmem + lanes + part * (HD / PT) + c + 8, o + 8);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(pready + (i & 1)));
        }
        // ---- the row's sum; then this thread's share of the dims
        s_part[nb & 1][part][r] = l;
        row_sync();
        l = s_part[nb & 1][0][r];
#pragma unroll
        for (int j = 1; j < PT; j++) l += s_part[nb & 1][j][r];
        if (nb > 0) {
            mbar_wait_reported(smem_u32(&ofull), 0, p.polls, p.err, 27);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        }
        if (DECODE && cs > 1) cluster_arrive_relaxed();                  // this CTA's MMAs are over
        pdl_wait();                                                      // (before the first store to memory)
        constexpr int DIMS = HD / PT, CH = DIMS < 32 ? DIMS : 32;
        if (DECODE && cs > 1) {
            // ---- partial state -> the blocks' shared memory, from where it is copied to the CTAs that finish the rows
            float* row = reinterpret_cast<float*>(smem + G::OUT) + r * G::OP;
            if (r < rows && part == 0) *reinterpret_cast<float2*>(row + HD) = make_float2(m, l);
            if (nb > 0) {
                uint32_t o[CH];
                tmem_ld<CH>(o, tmem + lanes + part * DIMS);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (r < rows) {
#pragma unroll
                    for (int j = 0; j < CH; j += 4) *reinterpret_cast<uint4*>(row + part * DIMS + j) = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        } else if (!DECODE && p.splits > 1) {
            // ---- partial state -> memory (of a range without keys: the merge multiplies it by zero)
            const size_t row = ((size_t)blockIdx.z * p.Hkv + hk) * p.n * p.G + (size_t)(ts * p.T + t) * p.G + g;
            if (valid && part == 0) *reinterpret_cast<float2*>(p.part_ml + row * 2) = make_float2(m, l);
#pragma unroll 1
            for (int c = part * DIMS; c < (part + 1) * DIMS; c += CH) {
                uint32_t o[CH] = {};
                if (nb > 0) tmem_ld<CH>(o, tmem + lanes + c);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (valid) {
#pragma unroll
                    for (int j = 0; j < CH; j += 4) *reinterpret_cast<uint4*>(p.part_o + row * HD + c + j) = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                }
            }
        } else {
            // ---- the whole row, through the queries' shared memory (their MMAs are over) so that stores cover whole rows
            const float inv = l > 0.f ? 1.f / l : 0.f;
            unsigned char* mine = smem + r * HD * 2;
#pragma unroll 1
            for (int c = part * DIMS; c < (part + 1) * DIMS; c += CH) {
                uint32_t o[CH] = {};
                if (nb > 0) tmem_ld<CH>(o, tmem + lanes + c);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < CH; j += 8) {
                    uint32_t h[4];
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        h[e] = h2_as_u32(__floats2half2_rn(__uint_as_float(o[j + 2 * e]) * inv, __uint_as_float(o[j + 2 * e + 1]) * inv));
                    *reinterpret_cast<uint4*>(mine + ((((c + j) >> 3) ^ (r & 7)) << 4)) = make_uint4(h[0], h[1], h[2], h[3]);
                }
            }
            row_sync();
            constexpr int V = HD / 8;                                    // 16-byte units of a row
#pragma unroll 4
            for (int k = part * 32 + lane; k < 32 * V; k += PT * 32) {
                const int rr = (warp & 3) * 32 + k / V, u = k % V, tt = rr / p.heads, gg = hs * p.heads + rr - tt * p.heads;
                if (rr < rows && gg < p.G)
                    *reinterpret_cast<uint4*>(p.out + ((size_t)(tok_base + tt) * p.Hq + hk * p.G + gg) * HD + u * 8) =
                        *reinterpret_cast<const uint4*>(smem + rr * HD * 2 + ((u ^ (rr & 7)) << 4));
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    }
    const bool row_warp = warp != G::LOADER && warp != G::ISSUER && (warp & 3) * 32 < rows;
    if (DECODE && cs > 1) {
        if (!row_warp) {
            if (warp != G::LOADER && warp != G::ISSUER) cluster_wait();  // (the peers have started: the others have waited)
            __syncwarp();
            cluster_arrive_relaxed();
        }
        cluster_wait();                                                  // the cluster's MMAs are over
    }
    __syncthreads();
    if (warp == G::ISSUER) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(kTmem) : "memory");
    }
    if (!DECODE || cs == 1) return;
    if (warp == G::LOADER && lane < (int)cs) {
        const int first = lane * nslot, n = min(nslot, rows - first);
        if (n > 0)
            bulk_copy_s2s(peer_addr(sbase + rank * nslot * G::OP * 4, lane), sbase + G::OUT + first * G::OP * 4, n * G::OP * 4, peer_addr(smem_u32(&inboxfull), lane));
    }
    // ---- merge: four dims of a row a thread, CTAs in key order
    inbox_wait(smem_u32(&inboxfull), p.polls, p.err, 25);
    __syncwarp();
    cluster_arrive_relaxed();                                            // what was copied here is here
#pragma unroll 1
    for (int k = threadIdx.x; k < mine_rows * (HD / 4); k += G::THREADS) {
        const int j = k / (HD / 4), c = (k % (HD / 4)) * 4;
        const float* src = reinterpret_cast<const float*>(smem) + j * G::OP;
        const int step = nslot * G::OP;
        float2 ml[8];
        float4 v[8];
        float mstar = -INFINITY;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            ml[i] = make_float2(-INFINITY, 0.f);
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < (int)cs) {
                ml[i] = *reinterpret_cast<const float2*>(src + i * step + HD);
                v[i] = *reinterpret_cast<const float4*>(src + i * step + c);
            }
            mstar = fmaxf(mstar, ml[i].x);
        }
        float den = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (ml[i].x != -INFINITY) {                                  // (a range without keys has left no output)
                const float w = exp2_approx(ml[i].x - mstar);
                den += w * ml[i].y;
                acc.x += w * v[i].x; acc.y += w * v[i].y; acc.z += w * v[i].z; acc.w += w * v[i].w;
            }
        const float inv = den > 0.f ? 1.f / den : 0.f;
        const int rr = row_lo + j, tt = rr / p.heads, gg = hs * p.heads + rr - tt * p.heads;
        if (gg < p.G)
            *reinterpret_cast<uint2*>(p.out + ((size_t)(tok_base + tt) * p.Hq + hk * p.G + gg) * HD + c) =
                make_uint2(h2_as_u32(__floats2half2_rn(acc.x * inv, acc.y * inv)), h2_as_u32(__floats2half2_rn(acc.z * inv, acc.w * inv)));
    }
    cluster_wait();                                                      // and what this CTA has copied from its memory is where it should be
}

template <int HD, bool DECODE>
int launch_flash(const FParams& f, dim3 grid, int cs, cudaStream_t stream) {
    using G = FGeo<HD, DECODE>;
    auto kern = flash_kernel<HD, DECODE>;
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(kern, G::SMEM, done, true)) return check_launch();
    return launch_chain(kern, grid, G::THREADS, G::SMEM, cs, stream, f);
}

FParams params(const FlashArgs& a, const FlashPlan& pl, int row0) {
    FParams f{};
    f.qmap = pl.qmap; f.kvmap = pl.kvmap;
    f.out = static_cast<__half*>(a.out);
    f.mask = a.mask; f.prefix = a.prefix; f.part_o = a.part_o; f.part_ml = a.part_ml;
    f.Hq = a.Hq; f.Hkv = a.Hkv; f.G = pl.G; f.heads = pl.heads; f.T = pl.T; f.hsets = pl.hsets; f.cap = a.cap; f.row0 = row0;
    f.mr = a.mr; f.tail = a.tail; f.write_off = a.write_off; f.nkb = a.nkb; f.req_rows = a.req_rows;
    f.n = a.tokens; f.off = a.off; f.splits = a.splits;
    f.scale_log2 = a.scale_log2; f.err = a.err; f.polls = a.polls;
    return f;
}

// Boxes of `rows` query rows at most: whole groups of as many tokens as fit, or part of a wider group.
int maps(const FlashArgs& a, FlashPlan* p, int ntok, int rows) {
    p->G = a.Hq / a.Hkv;
    p->heads = std::min(p->G, rows);
    p->T = std::min(ntok, rows / p->heads);
    p->hsets = (p->G + p->heads - 1) / p->heads;
    p->tsets = (ntok + p->T - 1) / p->T;
    const uint64_t heads = (uint64_t)a.Hq + 2 * a.Hkv;
    int rc = make_map_3d(&p->qmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.q, a.hd, heads, a.tokens, (uint64_t)a.hd * 2, heads * a.hd * 2, 64, p->heads, p->T,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
    if (rc != B200_OK) return rc;
    return make_map_2d(&p->kvmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.kv, a.hd, a.kv_rows, (uint64_t)a.hd * 2, 64, kKeyBlock, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
}

}  // namespace

// Clusters of as many key ranges as still run at once, two CTAs to an SM (33 clusters of 8 fit, 71 of 4).  `split` as
// b200_forward_desc.attn_split_blocks.
int flash_decode_plan(const FlashArgs& a, FlashPlan* p) {
    const int rc = maps(a, p, a.mr, 64);
    if (rc != B200_OK) return rc;
    const int clusters = a.Hkv * p->hsets * p->tsets * a.nreq;
    int cs = std::min(a.nkb, 8);
    while (a.split >= 0 && cs > 1 && clusters > 8 * (32 / cs)) cs--;
    if (a.split > 0 && a.nkb < a.split) cs = 1;
    p->cs = cs;
    return B200_OK;
}

int flash_decode(const FlashArgs& a, const FlashPlan& p, int row0, cudaStream_t stream) {
    const FParams f = params(a, p, row0);
    const dim3 grid(p.cs, a.Hkv * p.hsets * p.tsets, a.nreq);
    return a.hd == 128 ? launch_flash<128, true>(f, grid, p.cs, stream) : launch_flash<64, true>(f, grid, p.cs, stream);
}

int flash_prefill_plan(const FlashArgs& a, FlashPlan* p) {
    p->cs = 1;
    return maps(a, p, a.tokens, 128);
}

int flash_prefill(const FlashArgs& a, const FlashPlan& p, int row0, cudaStream_t stream) {
    const FParams f = params(a, p, row0);
    const dim3 grid(p.hsets * p.tsets, a.Hkv, a.splits);
    return a.hd == 128 ? launch_flash<128, false>(f, grid, 1, stream) : launch_flash<64, false>(f, grid, 1, stream);
}

}  // namespace b200
