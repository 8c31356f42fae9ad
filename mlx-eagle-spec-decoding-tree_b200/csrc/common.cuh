// Shared device helpers for the sm_100a kernels of the tree speculative decoding path.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "b200_eagle.h"

namespace b200 {

// Last CUDA runtime error seen by any entry point of this library (per process).
extern int g_last_cuda_error;

inline int check_launch() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return B200_ECUDA;
    }
    return B200_OK;
}

// Programmatic dependent launch: every kernel of this library may start while its predecessor in
// the stream is still draining; it must execute pdl_wait() before it reads anything an earlier
// kernel wrote and before its first global write.  0 disables the launch attribute.
extern int g_use_pdl;

// Poll limit of the device-side waits, set by b200_set_wait_limit; 0 = each kernel's built-in default (seconds).
extern unsigned g_wait_limit;
extern std::atomic<unsigned> g_launch_settings;   // changes with each setting of the process

// Of a kernel whose own limit is `built_in` and which takes no more than `most`.
inline int wait_polls(uint32_t built_in, uint32_t most) { return (int)(g_wait_limit == 0 ? built_in : (g_wait_limit < most ? g_wait_limit : most)); }

template <typename... KArgs, typename... Args>
inline void launch_kernel(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// A kernel of the chain: programmatic dependent launch, clusters of `cluster` CTAs along x.
template <typename P>
int launch_chain(void (*kern)(P), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t stream, const P& p) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (g_use_pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        n++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, kern, p);
    return check_launch();
}

// Lets `kern` use `bytes` of dynamic shared memory: a per-device attribute, set once per device (`done`: one bit each, a static
// of the caller's).
// `whole`: prefer the largest shared-memory carve-out, for kernels meant to have two CTAs on an SM.
template <typename F>
inline bool allow_smem(F kern, size_t bytes, std::atomic<uint64_t>& done, bool whole = false) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return false;
    if (whole && cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess) return false;
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 u32_as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// D(16x8, fp32) += A(16x16, fp16, row) * B(16x8, fp16, col); the warp-level tensor-core op used
// for the skinny (<= 32 token) products of this path.
__device__ __forceinline__ void mma_m16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                             uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace b200
