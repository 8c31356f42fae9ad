// Prompt ingestion: one causal pass of many tokens, every layer's kernels launched from native code.
//
//   embedding + input norm | per layer: q|k|v matmul (+ bias) -> RoPE + KV append -> causal attention -> o_proj matmul
//   (+ residual) -> norm -> gate/up matmul (SiLU(gate) * up) -> down matmul (+ residual) -> norm | vocabulary projection
//
// The matmuls are csrc/qmm_gemm.cu and, beyond 128 tokens where it is cheaper, csrc/qmm_pair.cu, attention is csrc/flash.cu; the
// element-wise steps that do not fit their epilogues are the kernels below (8B shape, 1024 tokens: 17 of 420 us a layer; their waits hidden
// behind the matmul before them, nothing was gained: such a pass runs at the power limit).  Up to 128 tokens of a small model go
// through the matmuls of csrc/decode.cu instead, which RoPE and append themselves.  Rounding points are those of the 32-row path's
// per-op kernels either way: norm (fp32) -> fp16, product -> fp16, + bias / + residual in fp16, SiLU(gate) * up with fp16 results, probabilities -> fp16.
// Replaces the chunk loop of mlx_eagle.py:522-535 over mlx_llama.py:231-249.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "decode.cuh"
#include "flash.cuh"
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

// The same between the kernels of csrc/decode.cu, a row a CTA.  The next of them comes up and expands its first weights while this one
// waits, but for the first of a pass (FIRST: with `tokens`), which lets it go behind the wait, like embed_kernel there, and makes the
// tokens' rotations.  What bounds it: start, one load and code that runs for the first time, 1.2 us a norm (61 tokens of the 0.5B shape
// 660 -> 722 us with norms that the matmuls on both sides shared before, as in passes of up to 32 tokens, and whose products with h did not
// always fit fp16).  A warp a row, four rows a CTA: 796; norm weights asked for behind the wait: 754.
struct ChainNorm {
    __half* x;
    const __half* w;
    __half* y;
    int H;
    float eps;
    const int* tokens;
    const uint32_t* wq;
    const __half* sc;
    const __half* bi;
    int V;
    float2* cs;                    // [n][kCsPitch]
    const float* inv_freq;
    float scaling;
    int off, half_hd;
};
template <bool FIRST, int UNITS>                                  // UNITS: 16-byte units of a thread
__global__ void __launch_bounds__(kNormThreads) chain_norm_kernel(const ChainNorm p) {
    const int row = blockIdx.x, units = p.H / 8;
    __half* const xr = p.x + (size_t)row * p.H;
    uint4 v[UNITS], w[UNITS];
    auto weights = [&]() {
#pragma unroll
        for (int i = 0; i < UNITS; i++) {
            const int u = threadIdx.x + i * blockDim.x;
            w[i] = u < units ? __ldg(reinterpret_cast<const uint4*>(p.w + u * 8)) : make_uint4(0, 0, 0, 0);
        }
    };
    if (!FIRST) {
        pdl_launch_dependents();
        weights();                                               // (there before the pass)
    }
    pdl_wait();
    if (FIRST) {
        pdl_launch_dependents();
        weights();
        if ((int)threadIdx.x < p.half_hd) {
            float s, c;
            sincosf((p.scaling * p.inv_freq[threadIdx.x]) * (float)(p.off + row), &s, &c);
            p.cs[row * kCsPitch + threadIdx.x] = make_float2(c, s);
        }
    }
    const int tok = FIRST ? min(max(p.tokens[row], 0), p.V - 1) : 0;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < UNITS; i++) {
        const int u = threadIdx.x + i * blockDim.x;
        v[i] = make_uint4(0, 0, 0, 0);
        if (u < units) {
            if (FIRST) {
                const uint32_t pk = p.wq[(size_t)tok * units + u];
                const __half s = p.sc[(size_t)tok * (p.H / 64) + (u >> 3)], b = p.bi[(size_t)tok * (p.H / 64) + (u >> 3)];
                __half* o = reinterpret_cast<__half*>(&v[i]);
#pragma unroll
                for (int j = 0; j < 8; j++) o[j] = __hfma(__int2half_rn((int)((pk >> (4 * j)) & 0xfu)), s, b);
                *reinterpret_cast<uint4*>(xr + u * 8) = v[i];
            } else {
                v[i] = __ldcg(reinterpret_cast<const uint4*>(xr + u * 8));
            }
        }
    }
#pragma unroll
    for (int i = 0; i < UNITS; i++) {
        const __half2* h = reinterpret_cast<const __half2*>(&v[i]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(h[j]);
            ss += f.x * f.x + f.y * f.y;
        }
    }
    const float inv = rsqrtf(block_sum(ss) / (float)p.H + p.eps);
#pragma unroll
    for (int i = 0; i < UNITS; i++) {
        const int u = threadIdx.x + i * blockDim.x;
        const __half2* h = reinterpret_cast<const __half2*>(&v[i]);
        const __half2* g = reinterpret_cast<const __half2*>(&w[i]);
        __align__(16) __half2 o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(h[j]), gf = __half22float2(g[j]);
            o[j] = __floats2half2_rn((f.x * inv) * gf.x, (f.y * inv) * gf.y);
        }
        if (u < units) *reinterpret_cast<uint4*>(p.y + (size_t)row * p.H + u * 8) = *reinterpret_cast<const uint4*>(o);
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

// Partial softmax states of the key ranges -> output: one warp per query row, ranges in order.
template <int HD>
__global__ void __launch_bounds__(256) prefill_attention_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, __half* __restrict__ out, int n,
                                                                      int Hq, int Hkv, int splits) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int G = Hq / Hkv, QR = n * G;
    const int idx = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (idx >= QR * Hkv) return;
    const int hk = idx / QR, r = idx - hk * QR;
    constexpr int C = HD / 32;
    float mstar = -INFINITY;
    for (int s = 0; s < splits; s++) mstar = fmaxf(mstar, __ldcg(part_ml + (((size_t)s * Hkv + hk) * QR + r) * 2));
    float acc[C], den = 0.f;
#pragma unroll
    for (int c = 0; c < C; c++) acc[c] = 0.f;
    for (int s = 0; s < splits; s++) {
        const size_t at = ((size_t)s * Hkv + hk) * QR + r;
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(part_ml) + at);
        const float w = ml.x == -INFINITY ? 0.f : exp2f(ml.x - mstar);
        den += ml.y * w;
#pragma unroll
        for (int c = 0; c < C; c++) acc[c] += w * __ldcg(part_o + at * HD + lane * C + c);
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
    const int m = r / G;
    __half* d = out + (size_t)m * Hq * HD + (size_t)(hk * G + r - m * G) * HD + lane * C;
#pragma unroll
    for (int c = 0; c < C; c++) d[c] = __float2half_rn(acc[c] * inv);
}

int launch_attention(const FlashArgs& a, const FlashPlan& plan, int row0, cudaStream_t st) {
    const int rc = flash_prefill(a, plan, row0, st);
    if (rc != B200_OK || a.splits == 1) return rc;
    launch_kernel(a.hd == 128 ? prefill_attention_merge_kernel<128> : prefill_attention_merge_kernel<64>, dim3((a.tokens * a.Hq + 7) / 8), dim3(256), 0, st,
                  static_cast<const float*>(a.part_o), static_cast<const float*>(a.part_ml), static_cast<__half*>(a.out), a.tokens, a.Hq, a.Hkv, a.splits);
    return check_launch();
}

// The chain's kernels for prompts: clusters add up K without going through memory, but every tile of 32 tokens expands the weights for itself.
// Against chunks of weights (128 x 128) times token tiles a layer, large kernels and these, us: 0.5B shape (910 chunks) 33 tokens 839, 677; 64 861,
// 687; 128 972, 894.  1B (3712) 64 800, 663; 65 839, 820; 128 900, 978.  8 layers of 2856 chunks 64 374, 314; 96 398, 398; 128 425, 448.  4 layers
// of the 7B shape (14224) 64 325, 355.
constexpr int kChainPromptTokens = 128;
bool chain_prompt_wins(const b200_prefill_desc* d) {
    auto chunks = [](long long n, long long k) { return (n + 127) / 128 * (k / 128); };
    const int nq = d->n_heads * d->head_dim;
    const long long layer = chunks(nq + 2ll * d->n_kv_heads * d->head_dim, d->hidden) + chunks(d->hidden, nq) + chunks(2ll * d->intermediate, d->hidden) +
                            chunks(d->hidden, d->intermediate);
    return d->n <= kChainPromptTokens && layer * ((d->n + 31) / 32) <= 11200;
}
int norm_rows(const b200_prefill_desc* d, void* x, const void* w, void* y, int rows, bool embed, cudaStream_t st) {
    launch_kernel(norm_rows_kernel, dim3(rows), dim3(kNormThreads), 0, st, static_cast<__half*>(x), static_cast<const __half*>(w),
                  static_cast<__half*>(y), d->hidden, d->rms_eps, embed ? d->tokens : nullptr, d->embed_wq,
                  static_cast<const __half*>(d->embed_scales), static_cast<const __half*>(d->embed_biases), d->vocab);
    return check_launch();
}

int chain_norm(const b200_prefill_desc* d, const void* w, float2* cs, bool first, cudaStream_t st) {
    const ChainNorm p{static_cast<__half*>(d->h), static_cast<const __half*>(w), static_cast<__half*>(d->xn), d->hidden, d->rms_eps, d->tokens, d->embed_wq,
                      static_cast<const __half*>(d->embed_scales), static_cast<const __half*>(d->embed_biases), d->vocab, cs, d->inv_freq, d->rope_scaling, d->off,
                      d->head_dim / 2};
    const dim3 threads(d->hidden <= 1024 ? 128 : kNormThreads);
    if (d->hidden <= 8 * kNormThreads) launch_kernel(first ? chain_norm_kernel<true, 1> : chain_norm_kernel<false, 1>, dim3(d->n), threads, 0, st, p);
    else launch_kernel(first ? chain_norm_kernel<true, 4> : chain_norm_kernel<false, 4>, dim3(d->n), threads, 0, st, p);
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

    const size_t half = (size_t)d->n_kv_heads * d->cache_rows * hd;
    FlashArgs a{};
    a.q = d->qkv; a.kv = d->kv_cache; a.kv_rows = (uint64_t)d->n_layers * 2 * d->n_kv_heads * d->cache_rows;
    a.out = d->attn; a.tokens = n; a.off = d->off; a.Hq = d->n_heads; a.Hkv = d->n_kv_heads; a.hd = hd; a.cap = d->cache_rows;
    a.scale_log2 = d->attn_scale * kLog2e; a.err = ga.err; a.polls = wait_polls(kWaitPolls, kFirmPolls / 2);
    FlashPlan flash{};
    int rc = flash_prefill_plan(a, &flash);
    if (rc != B200_OK) return rc;
    // key ranges: while the (row tile, kv head) pairs leave SMs idle, at least four blocks each
    const int items = flash.tsets * flash.hsets * d->n_kv_heads;
    const int nblk = (d->off + n + kKeyBlock - 1) / kKeyBlock;
    a.splits = std::max(1, std::min({148 / items, nblk / 4, 16}));
    const size_t per_split = (size_t)d->n_heads * n * (hd + 2) * sizeof(float);
    const size_t rotations = (size_t)n * kCsPitch * sizeof(float2), chain = chain_prompt_wins(d) && rotations <= ga.partial_bytes ? rotations : 0;      // (ahead of the ranges' partial states)
    while (a.splits > 1 && chain + a.splits * per_split + 16 > ga.partial_bytes) a.splits--;
    a.part_ml = ga.partial ? static_cast<float*>(ga.partial) + chain / sizeof(float) : nullptr;
    a.part_o = a.part_ml ? a.part_ml + (((size_t)a.splits * d->n_heads * n * 2 + 3) & ~(size_t)3) : nullptr;

    // Few tokens of a small model: the matmuls and attention of the 32-row passes, whose kernels RoPE and append themselves.
    if (chain > 0) {
        struct Context {
            const b200_prefill_desc* d;
            float2* cs;
            const FlashArgs* a;
            const FlashPlan* plan;
            bool tree;
        } context{d, static_cast<float2*>(ga.partial), &a, &flash, n <= 64 && a.splits > 1};
        ChainPrompt c{};
        c.d = d; c.err = ga.err; c.cs = context.cs;
        if (context.tree) {                                        // key ranges by the CTAs of a cluster, merged in the same kernel
            a.nreq = 1; a.mr = a.tail = n; a.nkb = (d->cache_rows + kKeyBlock - 1) / kKeyBlock;
            if ((rc = flash_decode_plan(a, &flash)) != B200_OK) return rc;
        }
        c.norm = [](const void* p, const void* w, bool first, cudaStream_t stream) {
            const Context* x = static_cast<const Context*>(p);
            return chain_norm(x->d, w, x->cs, first, stream);
        };
        c.attention = [](const void* p, int row0, cudaStream_t stream) {
            const Context* x = static_cast<const Context*>(p);
            return x->tree ? flash_decode(*x->a, *x->plan, row0, stream) : launch_attention(*x->a, *x->plan, row0, stream);
        };
        c.context = &context;
        rc = chain_prompt(c, st);
    } else {
        rc = norm_rows(d, d->h, d->layers[6], d->xn, n, true, st);
        for (int l = 0; l < d->n_layers && rc == B200_OK; l++) {
            const void* const* L = d->layers + (size_t)l * 8;       // qkv, qkv bias, o, gate, up, down, input norm, post norm
            __half* kc = static_cast<__half*>(d->kv_cache) + (size_t)l * 2 * half;
            __half* vc = kc + half;
            rc = gemm(d->xn, L[0], nullptr, L[1], nullptr, d->qkv, n, nqkv, H, B200_EPI_NONE);
            if (rc != B200_OK) break;
            launch_kernel(rope_append_kernel, dim3(n), dim3(256), 0, st, static_cast<__half*>(d->qkv), d->inv_freq, d->rope_scaling, kc, vc, d->off,
                          d->n_heads, d->n_kv_heads, hd, d->cache_rows);
            if ((rc = check_launch()) != B200_OK) break;
            if ((rc = launch_attention(a, flash, l * 2 * d->n_kv_heads * d->cache_rows, st)) != B200_OK) break;
            if ((rc = gemm(d->attn, L[2], nullptr, nullptr, d->h, d->h, n, H, nq, B200_EPI_RESIDUAL)) != B200_OK) break;
            if ((rc = norm_rows(d, d->h, L[7], d->xn, n, false, st)) != B200_OK) break;
            if ((rc = gemm(d->xn, L[3], L[4], nullptr, nullptr, d->act, n, I, H, B200_EPI_SILU_MUL)) != B200_OK) break;
            if ((rc = gemm(d->act, L[5], nullptr, nullptr, d->h, d->h, n, H, I, B200_EPI_RESIDUAL)) != B200_OK) break;
            if (l + 1 < d->n_layers) rc = norm_rows(d, d->h, L[8 + 6], d->xn, n, false, st);
        }
    }
    if (rc != B200_OK || d->head_out == 0) return rc;
    const int rows = d->head_out == 1 ? n : 1;
    rc = norm_rows(d, static_cast<__half*>(d->h) + (size_t)(n - rows) * H, d->final_norm, d->xn, rows, false, st);
    if (rc != B200_OK) return rc;
    return gemm(d->xn, d->lm_head_tiled, nullptr, nullptr, nullptr, d->logits, rows, d->vocab, H, B200_EPI_NONE);
}

}  // extern "C"
