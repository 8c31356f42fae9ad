// Shared-memory ring plumbing used by the streaming kernels: mbarrier operations with bounded
// waits, bulk asynchronous copies (global -> shared, completion counted on an mbarrier) and the
// consumer-only named barrier.  No copy here uses cluster multicast.
#pragma once

#include "common.cuh"

namespace b200 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false if the phase did not complete within `polls`.  A poll that does not find the phase complete suspends the thread for up to about a
// microsecond, so the limit is a time limit.  (Without a suspend-time hint a complete phase is seen in 14 cycles and a
// suspended thread is back ~60 cycles after the arrival; with a hint the same two took 100 and 75 to 100 cycles.)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t polls) {
    for (uint32_t i = 0; i < polls; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
constexpr int kWaitPolls = 1 << 19;             // of a wait before it reports: half a second
constexpr int kFirmPolls = 8 * kWaitPolls;      // after which it is over all the same
constexpr int kNoReport = kFirmPolls;
// A wait that runs out of its polls sets the error word (kNoReport: there is none) and goes on, for some seconds in all: what it waits for
// comes, since it depends on nothing but copies, MMAs, kernels before this one and waits like it.  Nothing runs ahead of one: a ring
// whose one side does not wait goes round twice, the other side then waits for a phase that has passed, and a CTA that left early
// would be stored to by its cluster and written to by its copies.  So no caller looks at the outcome, and the loops stay
// warp-uniform, which keeps the operands of copies and MMAs in uniform registers (eight MMAs and two commits: 290 cycles instead of
// 560).  Not unrolled: a kernel of the chain mostly runs code for the first time, and every line of it costs (a flag in shared
// memory that let the CTA's other waits give up too: 10 us of the 490 of a 0.5B-shape pass).
__device__ __forceinline__ void mbar_wait_reported(uint32_t bar, uint32_t parity, int polls, int* err, int code) {
    bool ok = mbar_try_wait(bar, parity);
#pragma unroll 1
    for (int i = 0; !ok && i < kFirmPolls; i++) {
        ok = mbar_try_wait(bar, parity);
        if (i == polls) atomicCAS(err, 0, code);
    }
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
    return r;
}
// Ahead of the first arrival or store at a peer, behind mbarrier inits (with their fence) that the block has synchronised on: nothing
// else passes, so nothing else is waited for.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Phase 0 of a barrier that counts the bytes of the cluster's st.async into this CTA's shared memory; longer than the peers' own waits take.
// No acquire from the cluster: the bytes counted are in this SM's shared memory, where no cache stands before them, and making the rest of
// memory coherent between the SMs of a cluster took 0.3 us of every kernel.
__device__ __forceinline__ void inbox_wait(uint32_t bar, int polls, int* err, int code) {
    bool ok = false;
#pragma unroll 1
    for (int i = 0; !ok && i < 4 * kFirmPolls; i++) {
        ok = mbar_try_wait(bar, 0);
        if (i == 4 * polls) atomicCAS(err, 0, code);
    }
}

// One lane of a converged warp.  A branch on this keeps the compiler's knowledge that everything else is warp-uniform, so the
// descriptors and addresses of tcgen05.mma and of copies stay in uniform registers: an MMA issues every 19 cycles instead of
// every 45 behind `if (lane == 0)`.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Same copy with an L2 eviction policy (from make_evict_first_policy): data that is streamed once should not
// push the small re-used tensors (KV cache, activations) out of L2.
__device__ __forceinline__ uint64_t make_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint64_t make_evict_normal_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;\n" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void bulk_copy_g2s_hint(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar), "l"(policy)
                 : "memory");
}
// 2-D tiled TMA load: box at (x, y) of the tensor map -> shared memory.
__device__ __forceinline__ void tma_box(uint32_t dst, const void* tmap, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void consumer_sync(int nthreads) {       // named barrier 1: consumer warps only
    asm volatile("bar.sync 1, %0;\n" ::"r"(nthreads) : "memory");
}

}  // namespace b200
