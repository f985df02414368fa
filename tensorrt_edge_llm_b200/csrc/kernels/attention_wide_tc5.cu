// Paged GQA attention over prompt-size query blocks, head size 128: two 128-row query tiles share every K / V tile.
//
// A CTA owns (block of 2 x 128 / G query tokens of one sequence, KV head, KV split); rows of a tile stack the G query heads of a KV
// head on consecutive tokens (row = token * G + g).  Keys come 128 at a time (two 64-token pages or one of 128):
//   S_t = Q_t Kᵀ    tcgen05.mma, both operands in shared memory (TMA), S_t in TMEM columns [128 t, 128 t + 128)
//   softmax         a warpgroup per query tile, one row per thread; probabilities go back to TMEM as 16-bit pairs, over the scores
//   O_t += P_t V    tcgen05.mma with P_t read from TMEM, V as an MN-major operand straight from its page
// The issue order S0 S1 | PV0 S0' | PV1 S1' | ... keeps the tensor cores on one tile while the other tile's exponentials run.  What
// bounds it: 16 exponentials a cycle and SM against 16384 of them per 1024 cycles of MMA time, so both sides take about 2048 cycles per
// pair of tiles.  One 128-row tile with 64 keys at a time and probabilities through shared memory (the form that head size 64 still
// takes) left the tensor cores idle three quarters of the time: 8129 tokens, 32 heads: 994 us (545 TFLOP/s), here 470 us.
// Blocks are numbered from the end of the step: the longest rows of a causal prompt start first, and a step of many one-row sequences
// beside a prompt portion launches no empty CTAs (a grid of sequences x tiles of the longest one spent 150 us on those).
//
// Threads: warps 0-3 / 4-7 softmax of tile 0 / 1, warp 8 TMA, warp 9 MMA issue and TMEM, warps 10-11 idle.  TMEM: S0 | S1 | O0 | O1.  All waits bounded.
#include <type_traits>

#include "host_utils.h"
#include "tc5_common.cuh"

namespace telb {

struct AttnWideParams {
    void* out;                 // [T, Hq, 128] 16-bit
    float* ws_o;               // [splits, T, Hq, 128] fp32 (splits > 1)
    float* ws_lse;             // [splits, T, Hq] log2-domain log-sum-exp
    const int* q_start;
    const int* q_len;
    const int* past_len;
    const int* page_table;     // [N, max_pages]
    const int* tree_mask;      // [T, mask_words] or null
    int mask_words, max_pages, page_size;
    int hq, hkv, group, tq;    // group = hq / hkv, tq = 128 / group query tokens per tile
    int splits, total_tokens, num_seqs;
    int window;                // sliding window, 0 = none, -1 = every row sees every cached and new token
    float scale_log2;          // softmax scale * log2(e), positive
    int* status;
};

constexpr int kWideThreads = 384;          // three warpgroups; registers are handed from the third to the softmax ones: 2 x 128 x 208 + 128 x 72 <= 384 x 168
constexpr int kWideStages = 2;
constexpr int kWideTile = 128 * 128 * 2;            // bytes of a Q, K or V tile
constexpr int kWideSmem = (2 + 2 * kWideStages) * kWideTile + 1024 + 256;
constexpr float kWideRescale = 8.0f;                // log2 units by which the running maximum may lag behind

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 fma_x2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(*reinterpret_cast<uint64_t*>(&d))
        : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
    return d;
}
__device__ __forceinline__ float2 add_x2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(*reinterpret_cast<uint64_t*>(&d)) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
    return d;
}

// Block `want` of the step's blocks of `bt` query tokens, sequence by sequence; every warp finds it for itself.
__device__ __forceinline__ bool wide_find_block(const int* __restrict__ q_len, int num_seqs, int bt, int want, int lane, int& seq, int& block) {
    int base = 0;
    for (int s0 = 0; s0 < num_seqs; s0 += 32) {
        const int n = s0 + lane < num_seqs ? (max(q_len[s0 + lane], 0) + bt - 1) / bt : 0;
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t past = __ballot_sync(0xffffffffu, base + incl > want);
        if (past) {
            const int l = __ffs(past) - 1;
            seq = s0 + l;
            block = want - base - __shfl_sync(0xffffffffu, incl - n, l);
            return true;
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
    }
    return false;
}

template <typename T>
__global__ void __launch_bounds__(kWideThreads, 1)
attn_wide_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_kv, AttnWideParams p) {
    constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* s_q = smem;
    uint8_t* s_k = s_q + 2 * kWideTile;
    uint8_t* s_v = s_k + kWideStages * kWideTile;
    uint64_t* q_full = reinterpret_cast<uint64_t*>(s_v + kWideStages * kWideTile);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + kWideStages;
    uint64_t* v_full = k_empty + kWideStages;
    uint64_t* v_empty = v_full + kWideStages;
    uint64_t* s_full = v_empty + kWideStages;        // [tile] scores of the next K tile are in TMEM (and every earlier MMA is done)
    uint64_t* p_full = s_full + 2;                   // [tile] probabilities are in TMEM (128 arrivals)
    uint64_t* o_full = p_full + 2;                   // [tile] the last P V is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    pdl_wait();              // step metadata and Q / KV are produced by earlier kernels
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int split = blockIdx.x % p.splits;
    const int kvh = (blockIdx.x / p.splits) % p.hkv;
    const int nblocks = gridDim.x / (p.splits * p.hkv);
    int seq = 0, block = 0;
    if (!wide_find_block(p.q_len, p.num_seqs, 2 * p.tq, nblocks - 1 - (int)(blockIdx.x / (p.splits * p.hkv)), lane, seq, block)) return;

    const int qlen = p.q_len[seq];
    const int past = p.past_len[seq];
    const int qrow0 = p.q_start[seq];
    const int tok0 = block * 2 * p.tq;               // first query token of the block (within the sequence)
    const int ntq = tok0 + p.tq < qlen ? 2 : 1;      // query tiles that hold rows
    const int kv_end = past + ((p.tree_mask || p.window < 0) ? qlen : min(qlen, tok0 + 2 * p.tq));
    const int tile_lo = p.window > 0 ? max(0, past + tok0 - p.window + 1) / 128 : 0;
    const int tile_hi = (kv_end + 127) / 128;
    const int per = (tile_hi - tile_lo + p.splits - 1) / p.splits;
    const int j0 = tile_lo + split * per;
    const int ntiles = max(0, min(tile_hi, j0 + per) - j0);

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < kWideStages; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&s_full[t], 1);
            mbar_init(&p_full[t], 128);
            mbar_init(&o_full[t], 1);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tensormap(&tma_q);
        prefetch_tensormap(&tma_kv);
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents(); // after the allocation: a dependent that allocates ahead of its own wait must not take the columns first

    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 8) {
            // ------------------------------ producer ------------------------------
            if (lane == 0 && ntiles > 0) {
                mbar_expect_tx(q_full, ntq * kWideTile);
                for (int t = 0; t < ntq; ++t)
    #pragma unroll
                    for (int c = 0; c < 2; ++c)
                        tma_load_3d(s_q + t * kWideTile + c * 16384, &tma_q, q_full, c * 64, kvh * p.group, qrow0 + tok0 + t * p.tq);
                const int* table = p.page_table + (size_t)seq * p.max_pages;
                for (int j = 0; j < ntiles; ++j) {
                    const int stage = j % kWideStages;
                    const uint32_t ph = ((j / kWideStages) & 1) ^ 1;
                    int row[2];
    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        int pos = (j0 + j) * 128 + h * 64;
                        if (pos >= kv_end) pos -= 64;            // past the end: rows that the mask hides
                        const int page = table[pos / p.page_size];
                        row[h] = page < 0 ? -1 : (page * 2 * p.hkv + kvh) * p.page_size + pos % p.page_size;
                    }
                    // A page that a window has retired: its keys are hidden, but its values still enter P V, times zero.  The other half of the
                    // tile stands in for it, since page 0 holds whatever another sequence wrote.
                    if (row[0] < 0) row[0] = max(row[1], kvh * p.page_size);
                    if (row[1] < 0) row[1] = row[0];
                    if (!mbar_wait(&k_empty[stage], ph, abort_flag, p.status, kStatusProducerTimeout)) break;
                    mbar_expect_tx(&k_full[stage], kWideTile);
    #pragma unroll
                    for (int h = 0; h < 2; ++h)
    #pragma unroll
                        for (int c = 0; c < 2; ++c)
                            tma_load_2d(s_k + stage * kWideTile + c * 16384 + h * 8192, &tma_kv, &k_full[stage], c * 64, row[h]);
                    if (!mbar_wait(&v_empty[stage], ph, abort_flag, p.status, kStatusProducerTimeout)) break;
                    mbar_expect_tx(&v_full[stage], kWideTile);
    #pragma unroll
                    for (int h = 0; h < 2; ++h)
    #pragma unroll
                        for (int c = 0; c < 2; ++c)
                            tma_load_2d(s_v + stage * kWideTile + c * 16384 + h * 8192, &tma_kv, &v_full[stage], c * 64, row[h] + p.hkv * p.page_size);
                }
            }
        } else if (warp == 9) {
            // ------------------------------ MMA issuer ------------------------------
            if (lane == 0 && ntiles > 0) {
                const uint32_t idesc_s = idesc_f16(128, 128, kBf16);
                const uint32_t idesc_o = idesc_f16(128, 128, kBf16, false, true);
                auto issue_s = [&](int t, int stage) {
                    const uint64_t dq = smem_desc_sw128(s_q + t * kWideTile);
                    const uint64_t dk = smem_desc_sw128(s_k + stage * kWideTile);
    #pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const uint64_t off = (uint64_t)((k >> 2) * 16384 >> 4) + 2 * (k & 3);
                        umma_f16(tmem_base + t * 128, dq + off, dk + off, idesc_s, k > 0 ? 1u : 0u);
                    }
                    umma_commit(&s_full[t]);
                };
                bool ok = mbar_wait(q_full, 0, abort_flag, p.status, kStatusMmaTimeout) &&
                          mbar_wait(&k_full[0], 0, abort_flag, p.status, kStatusMmaTimeout);
                if (ok) {
                    tc_fence_after_sync();
                    for (int t = 0; t < ntq; ++t) issue_s(t, 0);
                    umma_commit(&k_empty[0]);
                }
                for (int j = 0; j < ntiles && ok; ++j) {
                    const int stage = j % kWideStages, next = (j + 1) % kWideStages;
                    const bool more = j + 1 < ntiles;
                    ok = mbar_wait(&v_full[stage], (j / kWideStages) & 1, abort_flag, p.status, kStatusMmaTimeout);
                    if (ok && more) ok = mbar_wait(&k_full[next], ((j + 1) / kWideStages) & 1, abort_flag, p.status, kStatusMmaTimeout);
                    if (!ok) break;
                    const uint64_t dv = smem_desc_sw128_mn(s_v + stage * kWideTile, 16384, 1024);
                    for (int t = 0; t < ntq && ok; ++t) {
                        ok = mbar_wait(&p_full[t], j & 1, abort_flag, p.status, kStatusMmaTimeout);
                        if (!ok) break;
                        tc_fence_after_sync();
    #pragma unroll
                        for (int k = 0; k < 8; ++k)
                            umma_f16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + k * 8, dv + (uint64_t)(k * 2048 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                        // the next scores overwrite the probabilities: MMAs of one thread run in order
                        if (more) issue_s(t, next);
                        else umma_commit(&o_full[t]);
                    }
                    if (!ok) break;
                    umma_commit(&v_empty[stage]);
                    if (more) umma_commit(&k_empty[next]);
                }
            }
        }
    } else if (warp < 4 * ntq) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        // ------------------------------ softmax / epilogue ------------------------------
        const int t = warp >> 2, quad = warp & 3;
        const int r = quad * 32 + lane;                 // MMA row == TMEM lane
        const int ti = r / p.group;                     // token within the tile
        const int g = r - ti * p.group;
        const int first = tok0 + t * p.tq;              // first token of the tile, within the sequence
        const int qi = first + ti;
        const bool row_valid = qi < qlen;
        const uint32_t quad_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        const uint32_t s_addr = quad_addr + t * 128, o_addr = quad_addr + 256 + t * 128;
        const int* mask_row = p.tree_mask ? p.tree_mask + (size_t)(qrow0 + min(qi, qlen - 1)) * p.mask_words : nullptr;
        const int last_vis = p.window < 0 ? past + qlen - 1 : past + min(qi, qlen - 1);       // last visible cache slot (no tree mask)
        const int first_vis = p.window > 0 ? past + qi - p.window + 1 : 0;
        float m_used = -INFINITY, l_sum = 0.f;
        bool ok = true;
        for (int j = 0; j < ntiles; ++j) {
            if (!mbar_wait(&s_full[t], j & 1, abort_flag, p.status, kStatusEpilogueTimeout)) { ok = false; break; }
            tc_fence_after_sync();
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld_x32(s_addr + c * 32, s[c]);
            tmem_ld_wait();
            const int c0 = (j0 + j) * 128;
            // tiles that every row of this query tile sees whole need no mask (most tiles of a long prompt)
            const bool whole = !mask_row && p.window <= 0 && c0 + 127 <= (p.window < 0 ? past + qlen - 1 : past + first);
            if (!whole) {
                if (mask_row) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        // columns below `past` are visible, the others as the row's bits say; a window cuts both
                        const int n0 = c0 + c * 32 - past;           // new-token index of the chunk's first column
                        uint32_t vis = 0;
                        if (n0 < qlen) {
                            if (n0 <= -32) {
                                vis = 0xffffffffu;
                            } else if (n0 < 0) {
                                vis = (1u << -n0) - 1u;
                                vis |= (uint32_t)mask_row[0] << -n0;
                            } else {
                                const int w = n0 >> 5, sh = n0 & 31;
                                vis = (uint32_t)mask_row[w] >> sh;
                                if (sh && w + 1 < p.mask_words) vis |= (uint32_t)mask_row[w + 1] << (32 - sh);
                            }
                            if (qlen - n0 < 32) vis &= (1u << (qlen - n0)) - 1u;
                        }
                        const int hidden = first_vis - (c0 + c * 32);        // columns of the chunk that lie before the window
                        if (hidden > 0) vis = hidden < 32 ? vis & (0xffffffffu << hidden) : 0u;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (!((vis >> i) & 1u)) s[c][i] = 0xff800000u;
                    }
                } else {
                    const int hi = last_vis - c0, lo = first_vis - c0;
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c * 32 + i > hi || c * 32 + i < lo) s[c][i] = 0xff800000u;
                }
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                mx[c] = __uint_as_float(s[c][0]);
#pragma unroll
                for (int i = 1; i < 31; i += 2) mx[c] = fmaxf(fmaxf(mx[c], __uint_as_float(s[c][i])), __uint_as_float(s[c][i + 1]));
                mx[c] = fmaxf(mx[c], __uint_as_float(s[c][31]));
            }
            const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
            if (j == 0) {
                m_used = m_new;
            } else {
                const bool need = m_new > m_used + kWideRescale;
                if (__any_sync(0xffffffffu, need)) {
                    // the scores' commit covers P V of the tile before: O is at rest
                    const float f = need ? ex2_approx(m_used - m_new) : 1.f;
#pragma unroll 1
                    for (int c = 0; c < 8; ++c) {
                        uint32_t o[16];
                        tmem_ld_x16(o_addr + c * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                        tmem_st_x16(o_addr + c * 16, o);
                    }
                    if (need) {
                        l_sum *= f;
                        m_used = m_new;
                    }
                }
            }
            const float mref = m_used == -INFINITY ? 0.f : m_used;
            const float2 sc = make_float2(p.scale_log2, p.scale_log2), mm = make_float2(-mref, -mref);
            float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t pk[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float2 e = fma_x2(make_float2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])), sc, mm);
                    e.x = ex2_approx(e.x);
                    e.y = ex2_approx(e.y);
                    if (i & 1) acc1 = add_x2(acc1, e);
                    else acc0 = add_x2(acc0, e);
                    pk[i] = Cvt<T>::pack2(e.x, e.y);
                }
                tmem_st_x16(s_addr + c * 16, pk);
            }
            l_sum += (acc0.x + acc0.y) + (acc1.x + acc1.y);
            tmem_st_wait();
            tc_fence_before_sync();
            mbar_arrive(&p_full[t]);
        }
        // ---- epilogue ----
        if (ok && ntiles > 0) ok = mbar_wait(&o_full[t], 0, abort_flag, p.status, kStatusEpilogueTimeout);
        if (ok) {
            tc_fence_after_sync();
            const size_t tok = (size_t)qrow0 + qi;
            const int head = kvh * p.group + g;
            const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                float v[32];
                if (ntiles > 0) {
                    uint32_t o[32];
                    tmem_ld_x32(o_addr + c * 32, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[i]) * inv;
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = 0.f;
                }
                if (!row_valid) continue;
                if (p.splits == 1) {
                    T* dst = reinterpret_cast<T*>(p.out) + (tok * p.hq + head) * 128 + c * 32;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        uint4 u;
                        u.x = Cvt<T>::pack2(v[q * 8 + 0], v[q * 8 + 1]);
                        u.y = Cvt<T>::pack2(v[q * 8 + 2], v[q * 8 + 3]);
                        u.z = Cvt<T>::pack2(v[q * 8 + 4], v[q * 8 + 5]);
                        u.w = Cvt<T>::pack2(v[q * 8 + 6], v[q * 8 + 7]);
                        reinterpret_cast<uint4*>(dst)[q] = u;
                    }
                } else {
                    float* dst = p.ws_o + (((size_t)split * p.total_tokens + tok) * p.hq + head) * 128 + c * 32;
#pragma unroll
                    for (int q = 0; q < 8; ++q) reinterpret_cast<float4*>(dst)[q] = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                }
            }
            if (row_valid && p.splits > 1)
                p.ws_lse[((size_t)split * p.total_tokens + tok) * p.hq + head] = l_sum > 0.f ? m_used + log2f(l_sum) : -INFINITY;
        }
    }

    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

template <typename T>
static int launch_wide(const CUtensorMap& tq, const CUtensorMap& tkv, const AttnWideParams& p, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attn_wide_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem);
        if (e != cudaSuccess) return fail("cudaFuncSetAttribute(attn_wide)", e);
        configured = true;
    }
    // no more blocks than whole ones and one remainder per sequence
    const long long blocks = p.total_tokens / (2 * p.tq) + p.num_seqs;
    TELB_LAUNCH("attn_wide_kernel", (attn_wide_kernel<T>), dim3((unsigned)(blocks * p.hkv * p.splits)), dim3(kWideThreads), kWideSmem, stream, tq, tkv, p);
    TELB_CHECK_LAUNCH("attn_wide_kernel");
    return 0;
}

}  // namespace telb

using namespace telb;

extern "C" int telb_attn_combine_dense(const float* ws_o, const float* ws_lse, void* out, int rows, int splits, int d, int is_bf16,
                                       cudaStream_t stream);

// Head size 128, positive scale, page size 64 or 128; the rest as telb_paged_attention.
extern "C" int telb_paged_attention_wide(const void* q, const void* kv_layer, void* out, const int* q_start, const int* q_len,
                                         const int* past_len, const int* page_table, const int* tree_mask, int mask_words, int num_seqs,
                                         int total_tokens, int num_pages, int max_pages, int page_size, int hq, int hkv, float scale,
                                         int window, int splits, float* ws, long long ws_floats, int is_bf16, int* status, cudaStream_t stream) {
    AttnWideParams p{};
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
    p.group = hq / hkv;
    p.tq = 128 / p.group;
    p.total_tokens = total_tokens;
    p.num_seqs = num_seqs;
    p.window = window;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.status = status;
    if (splits < 1) splits = 1;
    while (splits > 1 && (long long)splits * total_tokens * hq * 129 > ws_floats) --splits;
    p.splits = splits;
    p.ws_o = ws;
    p.ws_lse = ws ? ws + (size_t)splits * total_tokens * hq * 128 : nullptr;
    const CUtensorMapDataType dt = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap tq, tkv;
    const uint64_t dims[3] = {128, (uint64_t)hq, (uint64_t)total_tokens};
    const uint64_t strides[2] = {256, (uint64_t)hq * 256};
    const uint32_t box[3] = {64, (uint32_t)p.group, (uint32_t)p.tq};
    if (make_tmap_nd(&tq, dt, 3, q, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (make_tmap_2d(&tkv, dt, 2, kv_layer, (uint64_t)num_pages * 2 * hkv * page_size, 128, 256, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    const int rc = is_bf16 ? launch_wide<__nv_bfloat16>(tq, tkv, p, stream) : launch_wide<__half>(tq, tkv, p, stream);
    if (rc || splits == 1) return rc;
    return telb_attn_combine_dense(p.ws_o, p.ws_lse, out, total_tokens * hq, splits, 128, is_bf16, stream);
}
