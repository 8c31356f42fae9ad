// Prompt ingestion: one causal pass of many tokens, every layer's kernels launched from native code.
//
//   embedding + input norm | per layer: q|k|v matmul (+ bias) -> RoPE + KV append -> causal attention -> o_proj matmul
//   (+ residual) -> norm -> gate/up matmul (SiLU(gate) * up) -> down matmul (+ residual) -> norm | vocabulary projection
//
// The matmuls are csrc/qmm_gemm.cu (one weight read per 128 tokens, from L2 after the first); the element-wise steps that
// do not fit their epilogues are the kernels below.  Rounding points are those of the 32-row path's per-op kernels: norm ->
// fp16, product -> fp16, + bias / + residual in fp16, SiLU(gate) * up with fp16 results, probabilities -> fp16.
// Replaces the chunk loop of mlx_eagle.py:522-535 over mlx_llama.py:231-249.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "pipeline.cuh"
#include "qmm_common.cuh"
#include "qmm_gemm.cuh"

namespace b200 {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kKeyBlock = 64;

__device__ __forceinline__ float block_sum(float v) {
    __shared__ float red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += red[i];
    return s;
}

// y = fp16((x * rsqrt(mean(x^2) + eps)) * w): one row per CTA, the row stays in registers between the two passes over it
// (16-byte loads, H <= 8192).  With `tokens` the row is the dequantised embedding of tokens[row] and is also stored to x.
constexpr int kNormThreads = 256;
__global__ void __launch_bounds__(kNormThreads) norm_rows_kernel(__half* __restrict__ x, const __half* __restrict__ w, __half* __restrict__ y,
                                                                 int H, float eps, const int* __restrict__ tokens,
                                                                 const uint32_t* __restrict__ wq, const __half* __restrict__ sc,
                                                                 const __half* __restrict__ bi, int V) {
    pdl_wait();
    pdl_launch_dependents();
    const int row = blockIdx.x;
    const int units = H / 8;
    __half* xr = x + (size_t)row * H;
    uint4 v[4];
    float ss = 0.f;
    const int tok = tokens ? min(max(tokens[row], 0), V - 1) : 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int u = threadIdx.x + i * kNormThreads;
        if (u < units) {
            if (tokens) {
                const uint32_t pk = wq[(size_t)tok * units + u];
                const __half s = sc[(size_t)tok * (H / 64) + (u >> 3)], b = bi[(size_t)tok * (H / 64) + (u >> 3)];
                __half* o = reinterpret_cast<__half*>(&v[i]);
#pragma unroll
                for (int j = 0; j < 8; j++) o[j] = __hfma(__int2half_rn((int)((pk >> (4 * j)) & 0xfu)), s, b);
                *reinterpret_cast<uint4*>(xr + u * 8) = v[i];
            } else {
                v[i] = *reinterpret_cast<const uint4*>(xr + u * 8);
            }
            const __half2* h = reinterpret_cast<const __half2*>(&v[i]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(h[j]);
                ss += f.x * f.x + f.y * f.y;
            }
        }
    }
    const float inv = rsqrtf(block_sum(ss) / (float)H + eps);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int u = threadIdx.x + i * kNormThreads;
        if (u < units) {
            const uint4 wv = *reinterpret_cast<const uint4*>(w + u * 8);
            const __half2* h = reinterpret_cast<const __half2*>(&v[i]);
            const __half2* g = reinterpret_cast<const __half2*>(&wv);
            __align__(16) __half2 o[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __half22float2(h[j]), gf = __half22float2(g[j]);
                o[j] = __floats2half2_rn((f.x * inv) * gf.x, (f.y * inv) * gf.y);
            }
            *reinterpret_cast<uint4*>(y + (size_t)row * H + u * 8) = *reinterpret_cast<const uint4*>(o);
        }
    }
}

// RoPE of q (in place) and k, KV append: one token per CTA; its cos / sin are computed once for all heads.
__global__ void __launch_bounds__(256) rope_append_kernel(__half* __restrict__ qkv, const float* __restrict__ inv_freq, float scaling,
                                                          __half* __restrict__ kc, __half* __restrict__ vc, int off, int Hq, int Hkv,
                                                          int hd, int cap) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ float2 cs[64];
    const int m = blockIdx.x, row = off + m;
    if ((int)threadIdx.x < hd / 2) {
        const float theta = (scaling * inv_freq[threadIdx.x]) * (float)row;
        float s, c;
        sincosf(theta, &s, &c);
        cs[threadIdx.x] = make_float2(c, s);
    }
    __syncthreads();
    const int hv = hd / 16;                                  // vector pairs (i, i + hd/2) per head
    __half* base = qkv + (size_t)m * (Hq + 2 * Hkv) * hd;
    for (int i = threadIdx.x; i < (Hq + Hkv) * hv; i += blockDim.x) {
        const int head = i / hv, c0 = (i - head * hv) * 8;
        __half* p1 = base + (size_t)head * hd + c0;
        const uint4 a = *reinterpret_cast<const uint4*>(p1), b = *reinterpret_cast<const uint4*>(p1 + hd / 2);
        const __half* x1 = reinterpret_cast<const __half*>(&a);
        const __half* x2 = reinterpret_cast<const __half*>(&b);
        __align__(16) __half r1[8], r2[8];
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const float2 t = cs[c0 + e];
            const float f1 = __half2float(x1[e]), f2 = __half2float(x2[e]);
            r1[e] = __float2half_rn(f1 * t.x - f2 * t.y);
            r2[e] = __float2half_rn(f1 * t.y + f2 * t.x);
        }
        __half* dst = head < Hq ? p1 : kc + ((size_t)(head - Hq) * cap + row) * hd + c0;
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(r1);
        *reinterpret_cast<uint4*>(dst + hd / 2) = *reinterpret_cast<const uint4*>(r2);
    }
    const int vv = hd / 8;
    for (int i = threadIdx.x; i < Hkv * vv; i += blockDim.x) {
        const int head = i / vv, c0 = (i - head * vv) * 8;
        *reinterpret_cast<uint4*>(vc + ((size_t)head * cap + row) * hd + c0) =
            *reinterpret_cast<const uint4*>(base + (size_t)(Hq + Hkv + head) * hd + c0);
    }
}

// ---- causal attention of n new tokens over off + n cache rows, GQA
// CTA = (128 query rows of one kv head, key range); a query row is (token, head of the group), so the group's heads share
// every K/V block.  Eight warps of 16 rows; 64-key blocks of K and V through a two-stage cp.async ring (16-byte units
// swizzled by the row, conflict-free ldmatrix); scores and the running softmax in fp32, probabilities fp16, mma.sync.
// Bound by mma.sync at these sizes (a few per cent of a prompt pass; the matmuls have the rest).  Few tokens on a long cache
// leave CTAs to spare: the key range is then cut and the partial (max, sum, output) merged by a second kernel.
struct PAttn {
    const __half* q;
    int q_stride;                  // halves between tokens
    const __half* kc;              // [Hkv][cap][HD]
    const __half* vc;
    __half* out;                   // [n][Hq * HD]
    float* part_o;                 // [split][Hq * n rows][HD]
    float* part_ml;                // [split][Hq * n rows][2]
    int n, off, Hq, Hkv, cap, splits;
    float scale_log2;
};

constexpr int kPRows = 128;
__device__ __forceinline__ uint32_t pswz(int r, int u, int hd) { return (uint32_t)(r * hd * 2 + ((u ^ (r & 7)) << 4)); }

template <int HD>
__global__ void __launch_bounds__(256) prefill_attention_kernel(const PAttn p) {
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int BLK = kKeyBlock * HD * 2;               // bytes of a K (or V) block
    const uint32_t sbase = smem_u32(smem);
    const int G = p.Hq / p.Hkv;
    const int QR = p.n * G;
    const int tile = (int)gridDim.x - 1 - (int)blockIdx.x;      // the longest key ranges first
    const int hk = blockIdx.y, split = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int row_last = min(tile * kPRows + kPRows, QR) - 1;
    const int nblk_all = (p.off + row_last / G) / kKeyBlock + 1;
    const int per = (nblk_all + p.splits - 1) / p.splits;
    const int blk0 = split * per, blk1 = min(blk0 + per, nblk_all);
    const __half* kbase = p.kc + (size_t)hk * p.cap * HD;
    const __half* vbase = p.vc + (size_t)hk * p.cap * HD;
    const int total = p.off + p.n;

    const int rw = tile * kPRows + warp * 16;                   // first row of the warp
    const int r0 = rw + g, r1 = r0 + 8;
    const bool v0 = r0 < QR, v1 = r1 < QR;
    const int m0 = v0 ? r0 / G : 0, m1 = v1 ? r1 / G : 0;
    const int lim0 = v0 ? p.off + m0 : -1, lim1 = v1 ? p.off + m1 : -1;       // last visible key
    const int wfirst = p.off + rw / G;                          // keys up to here are visible to every row of the warp
    const int wlast = rw < QR ? p.off + (min(rw + 15, QR - 1)) / G : -1;

    uint32_t qa[HD / 16][4];
    {
        const __half* q0 = p.q + (size_t)m0 * p.q_stride + (size_t)(hk * G + (v0 ? r0 - m0 * G : 0)) * HD;
        const __half* q1 = p.q + (size_t)m1 * p.q_stride + (size_t)(hk * G + (v1 ? r1 - m1 * G : 0)) * HD;
#pragma unroll
        for (int ks = 0; ks < HD / 16; ks++) {
            qa[ks][0] = *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 2 * t);
            qa[ks][1] = *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 2 * t);
            qa[ks][2] = *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 2 * t + 8);
            qa[ks][3] = *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 2 * t + 8);
        }
    }
    auto load = [&](int b) {
        const uint32_t s = sbase + (b & 1) * 2 * BLK;
        constexpr int VPR = HD / 8;
#pragma unroll
        for (int i = threadIdx.x; i < kKeyBlock * VPR; i += 256) {
            const int r = i / VPR, u = i - r * VPR;
            const int key = min(b * kKeyBlock + r, total - 1);          // rows past the end are masked; read a valid one
            cp_async16(s + pswz(r, u, HD), kbase + (size_t)key * HD + u * 8);
            cp_async16(s + BLK + pswz(r, u, HD), vbase + (size_t)key * HD + u * 8);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float mrun0 = -INFINITY, mrun1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    float o[HD / 8][4];
#pragma unroll
    for (int nd = 0; nd < HD / 8; nd++) o[nd][0] = o[nd][1] = o[nd][2] = o[nd][3] = 0.f;

    if (blk0 < blk1) load(blk0);
    for (int b = blk0; b < blk1; b++) {
        if (b + 1 < blk1) {
            load(b + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const int key0 = b * kKeyBlock;
        if (key0 <= wlast) {
            const uint32_t sk = sbase + (b & 1) * 2 * BLK, sv = sk + BLK;
            float s[8][4];
#pragma unroll
            for (int nt = 0; nt < 8; nt++) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
            for (int ks = 0; ks < HD / 16; ks += 2) {
#pragma unroll
                for (int nt = 0; nt < 8; nt++) {
                    uint32_t kf[4];
                    ldsm4(kf, sk + pswz(nt * 8 + (lane & 7), ks * 2 + (lane >> 3), HD));
                    mma_m16n8k16(s[nt], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], kf[0], kf[1]);
                    mma_m16n8k16(s[nt], qa[ks + 1][0], qa[ks + 1][1], qa[ks + 1][2], qa[ks + 1][3], kf[2], kf[3]);
                }
            }
            float mx0 = mrun0, mx1 = mrun1;
            if (key0 + kKeyBlock - 1 <= wfirst && rw + 15 < QR) {
#pragma unroll
                for (int nt = 0; nt < 8; nt++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        s[nt][e] *= p.scale_log2;
                        s[nt][2 + e] *= p.scale_log2;
                        mx0 = fmaxf(mx0, s[nt][e]);
                        mx1 = fmaxf(mx1, s[nt][2 + e]);
                    }
            } else {
#pragma unroll
                for (int nt = 0; nt < 8; nt++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int key = key0 + nt * 8 + 2 * t + e;
                        s[nt][e] = key <= lim0 ? s[nt][e] * p.scale_log2 : -INFINITY;
                        s[nt][2 + e] = key <= lim1 ? s[nt][2 + e] * p.scale_log2 : -INFINITY;
                        mx0 = fmaxf(mx0, s[nt][e]);
                        mx1 = fmaxf(mx1, s[nt][2 + e]);
                    }
            }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            const float base0 = (mx0 == -INFINITY) ? 0.f : mx0;
            const float base1 = (mx1 == -INFINITY) ? 0.f : mx1;
            if (mx0 != mrun0 || mx1 != mrun1) {
                const float al0 = (mrun0 == -INFINITY) ? 0.f : exp2f(mrun0 - base0);
                const float al1 = (mrun1 == -INFINITY) ? 0.f : exp2f(mrun1 - base1);
                mrun0 = mx0; mrun1 = mx1;
                l0 *= al0; l1 *= al1;
#pragma unroll
                for (int nd = 0; nd < HD / 8; nd++) { o[nd][0] *= al0; o[nd][1] *= al0; o[nd][2] *= al1; o[nd][3] *= al1; }
            }
            uint32_t pa[8][2];
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
                const __half2 h0 = __floats2half2_rn(exp2f(s[nt][0] - base0), exp2f(s[nt][1] - base0));
                const __half2 h1 = __floats2half2_rn(exp2f(s[nt][2] - base1), exp2f(s[nt][3] - base1));
                // the sum uses the rounded probabilities so that numerator and denominator agree
                l0 += __low2float(h0) + __high2float(h0);
                l1 += __low2float(h1) + __high2float(h1);
                pa[nt][0] = h2_as_u32(h0);
                pa[nt][1] = h2_as_u32(h1);
            }
#pragma unroll
            for (int kk = 0; kk < kKeyBlock / 16; kk++) {
#pragma unroll
                for (int nd = 0; nd < HD / 8; nd += 2) {
                    uint32_t vb[4];
                    ldsm4_t(vb, sv + pswz(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), nd + (lane >> 4), HD));
                    mma_m16n8k16(o[nd], pa[2 * kk][0], pa[2 * kk][1], pa[2 * kk + 1][0], pa[2 * kk + 1][1], vb[0], vb[1]);
                    mma_m16n8k16(o[nd + 1], pa[2 * kk][0], pa[2 * kk][1], pa[2 * kk + 1][0], pa[2 * kk + 1][1], vb[2], vb[3]);
                }
            }
        }
        __syncthreads();                                        // the stage is refilled next
    }
    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
    if (p.splits > 1) {
        float* po = p.part_o + ((size_t)split * p.Hkv + hk) * QR * HD;
        float* pml = p.part_ml + ((size_t)split * p.Hkv + hk) * QR * 2;
        if (v0) {
            if (t == 0) *reinterpret_cast<float2*>(pml + (size_t)r0 * 2) = make_float2(mrun0, l0);
#pragma unroll
            for (int nd = 0; nd < HD / 8; nd++) *reinterpret_cast<float2*>(po + (size_t)r0 * HD + nd * 8 + 2 * t) = make_float2(o[nd][0], o[nd][1]);
        }
        if (v1) {
            if (t == 0) *reinterpret_cast<float2*>(pml + (size_t)r1 * 2) = make_float2(mrun1, l1);
#pragma unroll
            for (int nd = 0; nd < HD / 8; nd++) *reinterpret_cast<float2*>(po + (size_t)r1 * HD + nd * 8 + 2 * t) = make_float2(o[nd][2], o[nd][3]);
        }
        return;
    }
    const float i0 = l0 > 0.f ? 1.f / l0 : 0.f, i1 = l1 > 0.f ? 1.f / l1 : 0.f;
    __half* d0 = p.out + (size_t)m0 * p.Hq * HD + (size_t)(hk * G + (v0 ? r0 - m0 * G : 0)) * HD;
    __half* d1 = p.out + (size_t)m1 * p.Hq * HD + (size_t)(hk * G + (v1 ? r1 - m1 * G : 0)) * HD;
#pragma unroll
    for (int nd = 0; nd < HD / 8; nd++) {
        if (v0) *reinterpret_cast<__half2*>(d0 + nd * 8 + 2 * t) = __floats2half2_rn(o[nd][0] * i0, o[nd][1] * i0);
        if (v1) *reinterpret_cast<__half2*>(d1 + nd * 8 + 2 * t) = __floats2half2_rn(o[nd][2] * i1, o[nd][3] * i1);
    }
}

// Partial softmax states of the key ranges -> output: one warp per query row, ranges in order.
template <int HD>
__global__ void __launch_bounds__(256) prefill_attention_merge_kernel(const PAttn p) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int G = p.Hq / p.Hkv, QR = p.n * G;
    const int idx = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (idx >= QR * p.Hkv) return;
    const int hk = idx / QR, r = idx - hk * QR;
    constexpr int C = HD / 32;
    float mstar = -INFINITY;
    for (int s = 0; s < p.splits; s++) mstar = fmaxf(mstar, __ldcg(p.part_ml + (((size_t)s * p.Hkv + hk) * QR + r) * 2));
    float acc[C], den = 0.f;
#pragma unroll
    for (int c = 0; c < C; c++) acc[c] = 0.f;
    for (int s = 0; s < p.splits; s++) {
        const size_t at = ((size_t)s * p.Hkv + hk) * QR + r;
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml) + at);
        const float w = ml.x == -INFINITY ? 0.f : exp2f(ml.x - mstar);
        den += ml.y * w;
#pragma unroll
        for (int c = 0; c < C; c++) acc[c] += w * __ldcg(p.part_o + at * HD + lane * C + c);
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    const int m = r / G;
    __half* d = p.out + (size_t)m * p.Hq * HD + (size_t)(hk * G + r - m * G) * HD + lane * C;
#pragma unroll
    for (int c = 0; c < C; c++) d[c] = __float2half_rn(acc[c] * inv);
}

template <int HD>
int launch_attention(const PAttn& a, cudaStream_t st) {
    constexpr size_t smem = (size_t)4 * kKeyBlock * HD * 2;
    static std::atomic<uint64_t> done{0};
    if (!allow_smem(prefill_attention_kernel<HD>, smem, done)) return check_launch();
    const int QR = a.n * (a.Hq / a.Hkv);
    launch_kernel(prefill_attention_kernel<HD>, dim3((QR + kPRows - 1) / kPRows, a.Hkv, a.splits), dim3(256), smem, st, a);
    if (a.splits > 1)
        launch_kernel(prefill_attention_merge_kernel<HD>, dim3((QR * a.Hkv + 7) / 8), dim3(256), 0, st, a);
    return check_launch();
}

int norm_rows(const b200_prefill_desc* d, void* x, const void* w, void* y, int rows, bool embed, cudaStream_t st) {
    launch_kernel(norm_rows_kernel, dim3(rows), dim3(kNormThreads), 0, st, static_cast<__half*>(x), static_cast<const __half*>(w),
                  static_cast<__half*>(y), d->hidden, d->rms_eps, embed ? d->tokens : nullptr, d->embed_wq,
                  static_cast<const __half*>(d->embed_scales), static_cast<const __half*>(d->embed_biases), d->vocab);
    return check_launch();
}

}  // namespace
}  // namespace b200

extern "C" {

using namespace b200;

int b200_prefill(const b200_prefill_desc* d, void* stream) {
    if (!d || d->n < 1 || d->off < 0 || d->cache_rows < d->off + d->n || d->n_layers < 1 || d->n_heads < 1 || d->n_kv_heads < 1 ||
        d->n_heads % d->n_kv_heads || d->vocab < 8 || d->vocab % 8 || d->hidden < 128 || d->hidden % 128 || d->hidden > 8192 ||
        d->intermediate < 128 || d->intermediate % 128 || (d->n_heads * d->head_dim) % 128 || d->head_out < 0 || d->head_out > 2)
        return B200_EINVAL;
    if (d->head_dim != 64 && d->head_dim != 128) return B200_EUNSUPPORTED;
    const void* need[] = {d->tokens, d->inv_freq, d->embed_wq, d->embed_scales, d->embed_biases, d->final_norm, d->lm_head_tiled, d->layers,
                          d->h, d->xn, d->qkv, d->attn, d->act, d->kv_cache, d->workspace};
    for (const void* q : need)
        if (!q) return B200_EINVAL;
    if (d->head_out && !d->logits) return B200_EINVAL;
    const void* al[] = {d->final_norm, d->lm_head_tiled, d->h, d->xn, d->qkv, d->attn, d->act, d->kv_cache, d->workspace, d->logits};
    for (const void* q : al)
        if (!aligned16(q)) return B200_EALIGN;
    if (d->workspace_bytes < (size_t)kCounterBytes) return B200_EWORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int n = d->n, H = d->hidden, I = d->intermediate, hd = d->head_dim;
    const int nq = d->n_heads * hd, nqkv = (d->n_heads + 2 * d->n_kv_heads) * hd;

    GemmArgs ga{};
    ga.M = n;
    gemm_workspace(ga, d->workspace, d->workspace_bytes);
    auto gemm = [&](const void* x, const void* w, const void* w2, const void* bias, const void* extra, void* y, int rows, int N, int K, int epi) {
        ga.x = x; ga.w_tiled = w; ga.w2_tiled = w2; ga.bias = bias; ga.extra = extra; ga.y = y;
        ga.M = rows; ga.N = N; ga.K = K; ga.epilogue = epi;
        return qmm_gemm(ga, st);
    };

    PAttn a{};
    a.q = static_cast<const __half*>(d->qkv);
    a.q_stride = nqkv;
    a.out = static_cast<__half*>(d->attn);
    a.n = n; a.off = d->off; a.Hq = d->n_heads; a.Hkv = d->n_kv_heads; a.cap = d->cache_rows;
    a.scale_log2 = d->attn_scale * kLog2e;
    // key ranges: while the (row tile, kv head) pairs leave SMs idle, at least four blocks each
    const int G = d->n_heads / d->n_kv_heads;
    const int items = ((n * G + kPRows - 1) / kPRows) * d->n_kv_heads;
    const int nblk = (d->off + n + kKeyBlock - 1) / kKeyBlock;
    a.splits = std::max(1, std::min({148 / items, nblk / 4, 16}));
    const size_t per_split = (size_t)d->n_heads * n * (hd + 2) * sizeof(float);
    while (a.splits > 1 && a.splits * per_split > ga.partial_bytes) a.splits--;
    a.part_ml = static_cast<float*>(ga.partial);
    a.part_o = a.part_ml ? a.part_ml + (size_t)a.splits * d->n_heads * n * 2 : nullptr;
    const size_t half = (size_t)d->n_kv_heads * d->cache_rows * hd;

    int rc = norm_rows(d, d->h, d->layers[6], d->xn, n, true, st);
    for (int l = 0; l < d->n_layers && rc == B200_OK; l++) {
        const void* const* L = d->layers + (size_t)l * 8;       // qkv, qkv bias, o, gate, up, down, input norm, post norm
        __half* kc = static_cast<__half*>(d->kv_cache) + (size_t)l * 2 * half;
        __half* vc = kc + half;
        rc = gemm(d->xn, L[0], nullptr, L[1], nullptr, d->qkv, n, nqkv, H, B200_EPI_NONE);
        if (rc != B200_OK) break;
        launch_kernel(rope_append_kernel, dim3(n), dim3(256), 0, st, static_cast<__half*>(d->qkv), d->inv_freq, d->rope_scaling, kc, vc, d->off,
                      d->n_heads, d->n_kv_heads, hd, d->cache_rows);
        if ((rc = check_launch()) != B200_OK) break;
        a.kc = kc; a.vc = vc;
        if ((rc = hd == 128 ? launch_attention<128>(a, st) : launch_attention<64>(a, st)) != B200_OK) break;
        if ((rc = gemm(d->attn, L[2], nullptr, nullptr, d->h, d->h, n, H, nq, B200_EPI_RESIDUAL)) != B200_OK) break;
        if ((rc = norm_rows(d, d->h, L[7], d->xn, n, false, st)) != B200_OK) break;
        if ((rc = gemm(d->xn, L[3], L[4], nullptr, nullptr, d->act, n, I, H, B200_EPI_SILU_MUL)) != B200_OK) break;
        if ((rc = gemm(d->act, L[5], nullptr, nullptr, d->h, d->h, n, H, I, B200_EPI_RESIDUAL)) != B200_OK) break;
        if (l + 1 < d->n_layers) rc = norm_rows(d, d->h, L[8 + 6], d->xn, n, false, st);
    }
    if (rc != B200_OK || d->head_out == 0) return rc;
    const int rows = d->head_out == 1 ? n : 1;
    rc = norm_rows(d, static_cast<__half*>(d->h) + (size_t)(n - rows) * H, d->final_norm, d->xn, rows, false, st);
    if (rc != B200_OK) return rc;
    return gemm(d->xn, d->lm_head_tiled, nullptr, nullptr, nullptr, d->logits, rows, d->vocab, H, B200_EPI_NONE);
}

}  // extern "C"
