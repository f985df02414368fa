// Paged GQA attention on tcgen05: one kernel family for prefill chunks, decode rows and
// speculative tree verification.
//
// A CTA owns (sequence, KV head, 128-row query tile, KV split).  The 128 MMA rows stack the G
// query heads that share the KV head on top of 128/G consecutive query tokens (row = token*G + g),
// so a decode step (1 token) and a 60-token verification tree use the same tile shape as a
// prefill chunk and every K/V page is fetched once per KV head, not once per query head.
//   S = Q Kᵀ   tcgen05.mma, Q and K tiles in 128B-swizzled shared memory (TMA), S in TMEM (2 buffers)
//   softmax    4 warps, one row per thread, online max/sum with lazy rescaling of O (only when the
//              running max grows by more than 2^8), probabilities written to shared memory as bf16
//   O += P V   tcgen05.mma with V as an MN-major operand straight from the paged pool
// KV pages are 64 tokens (or 128, consumed as two 64-token tiles); the cache layer layout is
// [pages, 2, Hkv, P, D] so a (page, K|V, head) tile is one contiguous box for TMA.
// With `splits > 1` (decode at small batch) each split writes a normalised fp32 partial and its
// log-sum-exp to a workspace and `attn_combine_kernel` merges them.
//
// Roles (192 threads): warp 0 TMA producer, warp 1 MMA issuer / TMEM owner, warps 2-5 softmax.
// All waits are bounded (tc5_common.cuh).
//
// Reference counterparts: CuTe-DSL FMHA (kernelSrcs/fmha_cutedsl_blackwell/fmha.py), CTM decode
// (kernelSrcs/fmha_decode_ctm/fmha_decode.py) and XQA (kernelSrcs/xqa/mha.cu); semantics follow
// unittests/support/references.h:29-37 (bottom-right aligned causal mask, GQA, sliding window).
#include <type_traits>

#include "host_utils.h"
#include "tc5_common.cuh"

namespace telb {

struct AttnParams {
    void* out;                 // [T, Hq, D] 16-bit
    float* ws_o;               // [splits, T, Hq, D] fp32 (splits > 1)
    float* ws_lse;             // [splits, T, Hq]    log2-domain log-sum-exp
    const int* q_start;        // [N+1]
    const int* q_len;          // [N]
    const int* past_len;       // [N]
    const int* page_table;     // [N, max_pages]
    const int* tree_mask;      // [T, mask_words] or null
    int mask_words;
    int max_pages, page_size;
    int hq, hkv, group;        // group = hq / hkv
    int tq;                    // query tokens per tile = 128 / group
    int splits;
    int total_tokens;
    int window;                // sliding window, 0 = none, -1 = no causal mask (every row sees every cached and new token)
    float scale_log2;          // softmax scale * log2(e)
    int out_bf16;
    int* status;
};

constexpr int kAttnThreads = 192;
constexpr int kKvTile = 64;
constexpr float kRescaleThreshold = 8.0f;   // log2 units

// KVS: depth of the K and V tile rings; MINB: CTAs resident per SM.  Two resident CTAs with single-stage rings let
// one CTA's MMAs run under the other's softmax; one CTA with deep rings prefetches further ahead.
#define TELB_ATTN_EXTRA 0
#define TELB_ATTN_KERNEL attn_tc5_kernel
#include "attention_tc5_kernel.inc"
#undef TELB_ATTN_KERNEL
#undef TELB_ATTN_EXTRA

// Merge split partials: out = Σ_s 2^(lse_s - max) O_s / Σ_s 2^(lse_s - max).
// One CTA of D threads per (token, head); splits (<= 32) are weighted by lanes of warp 0 first so
// the D-wide accumulation issues all of its loads independently.
template <int D, typename T>
__global__ void attn_combine_kernel(const float* __restrict__ ws_o, const float* __restrict__ ws_lse, T* __restrict__ out,
                                    int total_rows /* T*Hq */, int splits) {
    pdl_prologue();
    __shared__ float w[32];
    const int row = blockIdx.x;
    const int d = threadIdx.x;
    if (threadIdx.x < 32) {
        const float l = threadIdx.x < splits ? ws_lse[(size_t)threadIdx.x * total_rows + row] : -INFINITY;
        float mx = l;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float e = (l == -INFINITY) ? 0.f : exp2f(l - mx);
        float den = e;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        w[threadIdx.x] = den > 0.f ? e / den : 0.f;
    }
    __syncthreads();
    float acc = 0.f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) acc += w[s] * __ldcg(&ws_o[((size_t)s * total_rows + row) * D + d]);
    out[(size_t)row * D + d] = Cvt<T>::from_f(acc);
}

template <int D, typename T, int KVS, int MINB>
static int launch_attn_variant(const CUtensorMap& tq, const CUtensorMap& tkv, const AttnParams& p, int qtiles, int nseq,
                               cudaStream_t stream) {
    constexpr int smem = 128 * D * 2 + 2 * KVS * kKvTile * D * 2 + 2 * 128 * kKvTile * 2 + 1024 + 512;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attn_tc5_kernel<D, T, KVS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail("cudaFuncSetAttribute(attn_tc5)", e);
        configured = true;
    }
    dim3 grid(qtiles, p.hkv, nseq * p.splits);
    TELB_LAUNCH("attn_tc5_kernel", (attn_tc5_kernel<D, T, KVS, MINB>), dim3(grid), dim3(kAttnThreads), smem, stream, tq, tkv, p);
    TELB_CHECK_LAUNCH("attn_tc5_kernel");
    if (p.splits > 1) {
        const int rows = p.total_tokens * p.hq;
        TELB_LAUNCH("attn_combine_kernel", (attn_combine_kernel<D, T>), dim3(rows), dim3(D), 0, stream, p.ws_o, p.ws_lse, reinterpret_cast<T*>(p.out), rows, p.splits);
        TELB_CHECK_LAUNCH("attn_combine_kernel");
    }
    return 0;
}

static int g_attn_variant = 1;       // measured 4-8 % faster than the deep-ring variant on prefill shapes

template <int D, typename T>
static int launch_attn(const CUtensorMap& tq, const CUtensorMap& tkv, const AttnParams& p, int qtiles, int nseq, cudaStream_t stream) {
    if (g_attn_variant == 1) return launch_attn_variant<D, T, 1, 2>(tq, tkv, p, qtiles, nseq, stream);     // 2 CTAs / SM, single-stage rings
    return launch_attn_variant<D, T, 4, 1>(tq, tkv, p, qtiles, nseq, stream);                              // 1 CTA / SM, four-stage rings
}

}  // namespace telb

using namespace telb;

// Ring depth / residency variant of the tile attention kernel (0 or 1: see launch_attn); process-wide.
extern "C" int telb_set_attn_variant(int v) {
    if (v < 0 || v > 1) return fail("telb_set_attn_variant: variant must be 0 or 1");
    g_attn_variant = v;
    return 0;
}

// Merge `splits` partial results (ws_o [splits, rows, d] fp32, ws_lse [splits, rows]) into out [rows, d] for head_dim 64 / 128;
// telb_attn_combine (attention_tc5_extra.cu) is the public entry and adds head_dim 256.
extern "C" int telb_attn_combine_dense(const float* ws_o, const float* ws_lse, void* out, int rows, int splits, int d, int is_bf16,
                                 cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (d == 128) {
        if (is_bf16) TELB_LAUNCH("attn_combine_kernel", (attn_combine_kernel<128, __nv_bfloat16>), dim3(rows), dim3(128), 0, stream, ws_o, ws_lse, (__nv_bfloat16*)out, rows, splits);
        else TELB_LAUNCH("attn_combine_kernel", (attn_combine_kernel<128, __half>), dim3(rows), dim3(128), 0, stream, ws_o, ws_lse, (__half*)out, rows, splits);
    } else if (d == 64) {
        if (is_bf16) TELB_LAUNCH("attn_combine_kernel", (attn_combine_kernel<64, __nv_bfloat16>), dim3(rows), dim3(64), 0, stream, ws_o, ws_lse, (__nv_bfloat16*)out, rows, splits);
        else TELB_LAUNCH("attn_combine_kernel", (attn_combine_kernel<64, __half>), dim3(rows), dim3(64), 0, stream, ws_o, ws_lse, (__half*)out, rows, splits);
    } else {
        return fail("telb_attn_combine: head_dim must be 64 or 128");
    }
    TELB_CHECK_LAUNCH("attn_combine_kernel");
    return 0;
}

extern "C" int telb_paged_attention_wide(const void* q, const void* kv_layer, void* out, const int* q_start, const int* q_len,
                                         const int* past_len, const int* page_table, const int* tree_mask, int mask_words, int num_seqs,
                                         int total_tokens, int num_pages, int max_pages, int page_size, int hq, int hkv, float scale,
                                         int window, int splits, float* ws, long long ws_floats, int is_bf16, int* status, cudaStream_t stream);

// The dense path (head_dim 64 / 128, no sinks, no skip-softmax); the public entry point telb_paged_attention lives in
// attention_tc5_extra.cu and forwards here when a step needs none of the extras.  The plain kernel has a translation unit of
// its own on purpose: sharing one with the extra instantiations cost it 17 % (175 -> 202 us at 8 x 1024 tokens).
// q [T,Hq,D], kv_layer [pages,2,Hkv,P,D], out [T,Hq,D]; metadata as in the ragged step ABI.
// ws must hold splits*T*Hq*(D+1) floats when splits > 1 (pass splits = 1 to avoid scratch).
extern "C" int telb_paged_attention_dense(const void* q, const void* kv_layer, void* out, const int* q_start,
                                    const int* q_len, const int* past_len, const int* page_table,
                                    const int* tree_mask, int mask_words, int num_seqs, int total_tokens,
                                    int max_q_len, int num_pages, int max_pages, int page_size, int hq, int hkv, int d,
                                    float scale, int window, int splits, float* ws, long long ws_floats, int is_bf16,
                                    int* status, int wide, cudaStream_t stream) {
    if (num_seqs <= 0 || total_tokens <= 0) return 0;
    if (d != 64 && d != 128) return fail("telb_paged_attention: head_dim must be 64 or 128 on the dense path");
    if (page_size != 64 && page_size != 128) return fail("telb_paged_attention: page size must be 64 or 128");
    if (hq % hkv) return fail("telb_paged_attention: Hq must be a multiple of Hkv");
    const int group = hq / hkv;
    if (group > 128 || (128 % group)) return fail("telb_paged_attention: GQA ratio must divide 128");
    // heads of 128: two query tiles a CTA (attention_wide_tc5.cu); its maxima are taken before the scale, which has to be positive
    if (wide && d == 128 && scale > 0.f)
        return telb_paged_attention_wide(q, kv_layer, out, q_start, q_len, past_len, page_table, tree_mask, mask_words, num_seqs, total_tokens,
                                         num_pages, max_pages, page_size, hq, hkv, scale, window, splits, ws, ws_floats, is_bf16, status, stream);
    AttnParams p{};
    p.out = out;
    p.q_start = q_start;
    p.q_len = q_len;
    p.past_len = past_len;
    p.page_table = page_table;
    p.tree_mask = tree_mask;
    p.mask_words = mask_words;
    p.max_pages = max_pages;
    p.page_size = page_size;
    p.hq = hq;
    p.hkv = hkv;
    p.group = group;
    p.tq = 128 / group;
    p.total_tokens = total_tokens;
    p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.out_bf16 = is_bf16;
    p.status = status;
    if (splits < 1) splits = 1;
    while (splits > 1 && (long long)splits * total_tokens * hq * (d + 1) > ws_floats) --splits;
    p.splits = splits;
    p.ws_o = ws;
    p.ws_lse = ws ? ws + (size_t)splits * total_tokens * hq * d : nullptr;
    const int qtiles = (max_q_len + p.tq - 1) / p.tq;
    const CUtensorMapDataType dt = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap tq, tkv;
    {
        const uint64_t dims[3] = {(uint64_t)d, (uint64_t)hq, (uint64_t)total_tokens};
        const uint64_t strides[2] = {(uint64_t)d * 2, (uint64_t)hq * d * 2};
        const uint32_t box[3] = {64, (uint32_t)group, (uint32_t)p.tq};
        if (make_tmap_nd(&tq, dt, 3, q, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    }
    {
        const uint64_t rows = (uint64_t)num_pages * 2 * hkv * page_size;
        if (make_tmap_2d(&tkv, dt, 2, kv_layer, rows, d, (uint64_t)d * 2, kKvTile, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    }
    if (d == 128) {
        if (is_bf16) return launch_attn<128, __nv_bfloat16>(tq, tkv, p, qtiles, num_seqs, stream);
        return launch_attn<128, __half>(tq, tkv, p, qtiles, num_seqs, stream);
    }
    if (is_bf16) return launch_attn<64, __nv_bfloat16>(tq, tkv, p, qtiles, num_seqs, stream);
    return launch_attn<64, __half>(tq, tkv, p, qtiles, num_seqs, stream);
}
