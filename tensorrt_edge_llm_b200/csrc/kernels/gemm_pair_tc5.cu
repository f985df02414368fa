// 16-bit (bf16 / fp16) GEMM for prompt-size M on CTA pairs (`tcgen05.mma.cta_group::2`, 256 x 256 per pair):
//     out[M,N] = x[M,K] . w[N,K]^T (x alpha[N], + bias, + residual), fp32 accumulation in TMEM
//
// What bounds it: a single CTA with a 128 x 256 tile moves 48 KB into and as much out of its shared memory per 64-wide K step of 512
// cycles, which leaves the MMAs waiting for operands.  A pair needs 32 KB per CTA and step (its own 128 rows of x, half of the w tile;
// the tensor cores of both SMs read both halves).  8129 x 24576 x 4096: 1270 us single, 1035 us here (1581 TFLOP/s).
//
// Both CTAs run the same tile sequence.  Every load completes on the leader's "stage full" barrier; the leader issues all MMAs; stage
// release and "accumulator full" reach both CTAs through the multicast commit; "accumulator drained" comes back from the epilogue warps
// of the pair.  Two 256-column accumulators fill TMEM, so a tile is converted and stored under the next one's main loop.
// Roles (10 warps): 0 TMA producer, 1 MMA issuer (leader) / TMEM owner, 2-9 epilogue (two warps per lane quadrant, 128 columns each).
// Every wait is bounded.  No TMA load uses cluster multicast.
//
// SwiGLU form: w holds the gate rows and behind them the up rows [2 x F, K]; CTA 0 keeps 128 gate rows, CTA 1 the matching up rows, and
// the epilogue writes silu(gate) * up [M, F] with the roundings of the separate pass (16-bit product, 16-bit activation).
// Squared-ReLU form: relu(product)^2, rounded likewise.
#include "gemm_common.cuh"
#include "pair_common.cuh"

namespace telb {

enum : int { kPairPlain = 0, kPairSwiglu = 1, kPairRelu2 = 2 };

constexpr int kPairBN = 256;
constexpr int kPairEpiWarps = 8;
constexpr int kPairThreads = 32 * (2 + kPairEpiWarps);
constexpr int kPairStage = 2 * 128 * kBK * 2;       // 128 rows of x and 128 of w per CTA
constexpr int kPairStages = 6;
constexpr int kPairSmem = kPairStages * kPairStage + 1024 + 256;

__device__ __forceinline__ void umma_f16_2(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

struct PairTile {
    int a0, tb;            // first row of the pair's tile, column-tile index
};
__device__ __forceinline__ PairTile pair_tile(const GemmParams& p, int t) {
    const int per_group = kRasterGroup * p.tiles_b;
    const int group = t / per_group;
    const int within = t - group * per_group;
    const int gfirst = group * kRasterGroup;
    const int gsize = min(kRasterGroup, p.tiles_a - gfirst);
    return PairTile{(gfirst + within % gsize) * 256, within / gsize};
}

template <typename T, int EPI>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStage);
    uint64_t* empty_bar = full_bar + kPairStages;
    uint64_t* tfull_bar = empty_bar + kPairStages;
    uint64_t* tempty_bar = tfull_bar + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t crank = cluster_ctarank_w();
    const bool leader = crank == 0;
    const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
    const int total_tiles = p.tiles_a * p.tiles_b;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull_bar[s], 1);
            mbar_init(&tempty_bar[s], 2 * kPairEpiWarps);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tensormap(&tma_a);
        prefetch_tensormap(&tma_b);
    }
    if (warp == 1) {
        tmem_alloc2(tmem_slot, 512);
        tmem_relinquish2();
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_w();       // both CTAs' barriers and TMEM exist before anything crosses the pair
    tc_fence_after_sync();
    pdl_prologue();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- producer: this CTA's rows of x, its half of w ----------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = cid; t < total_tiles && ok; t += ncl) {
                const PairTile w = pair_tile(p, t);
                const int arow = w.a0 + (int)crank * 128;
                const int brow = EPI == kPairSwiglu ? w.tb * 128 + (int)crank * p.rows_b : w.tb * kPairBN + (int)crank * 128;
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kStatusProducerTimeout)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = smem + stage * kPairStage;
                    const uint32_t fb = cluster_addr_of(&full_bar[stage], 0);
                    if (leader) mbar_expect_tx(&full_bar[stage], 2 * kPairStage);
                    tma_load_2d_pair(sa, &tma_a, fb, kb * kBK, arow);
                    tma_load_2d_pair(sa + kATileBytes, &tma_b, fb, kb * kBK, brow);
                    if (++stage == kPairStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            // ---------------- MMA issuer ----------------
            const uint32_t idesc = idesc_f16(256, kPairBN, p.out_bf16 != 0);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int i = 0;
            for (int t = cid; t < total_tiles && ok; t += ncl, ++i) {
                const int acc = i & 1;
                if (!mbar_wait(&tempty_bar[acc], ((uint32_t)(i >> 1) & 1u) ^ 1, abort_flag, p.status, kStatusMmaTimeout)) break;
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * kPairBN;
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, kStatusMmaTimeout)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint64_t da = smem_desc_sw128(smem + stage * kPairStage);
                    const uint64_t db = smem_desc_sw128(smem + stage * kPairStage + kATileBytes);
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) umma_f16_2(d_tmem, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit2(&empty_bar[stage], 3);
                    if (++stage == kPairStages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit2(&tfull_bar[acc], 3);
            }
        }
    } else {
        // ---------------- epilogue: lane quadrant `quad`, column half `grp` ----------------
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        int i = 0;
        for (int t = cid; t < total_tiles; t += ncl, ++i) {
            const PairTile w = pair_tile(p, t);
            const int acc = i & 1;
            if (!mbar_wait(&tfull_bar[acc], (uint32_t)(i >> 1) & 1u, abort_flag, p.status, kStatusEpilogueTimeout)) break;
            tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * kPairBN;
            const int row = w.a0 + (int)crank * 128 + quad * 32 + lane;
            const bool row_ok = row < p.rows_a;
            if constexpr (EPI == kPairSwiglu) {
#pragma unroll 1
                for (int c = 0; c < 2; ++c) {
                    const int f0 = grp * 64 + c * 32;
                    uint32_t rg[32], ru[32];
                    tmem_ld_x32(t_addr + f0, rg);
                    tmem_ld_x32(t_addr + 128 + f0, ru);
                    tmem_ld_wait();
                    const int col0 = w.tb * 128 + f0;
                    const int nvalid = min(32, p.rows_b - col0);
                    if (row_ok && nvalid > 0) {
                        float v[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            const float g = Cvt<T>::to_f(Cvt<T>::from_f(__uint_as_float(rg[j]))), u = Cvt<T>::to_f(Cvt<T>::from_f(__uint_as_float(ru[j])));
                            v[j] = g / (1.f + __expf(-g)) * u;
                        }
                        epilogue_store<T>(p, v, row, col0, nvalid);
                    }
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_x32(t_addr + grp * 128 + c * 32, r);
                    tmem_ld_wait();
                    const int col0 = w.tb * kPairBN + grp * 128 + c * 32;
                    const int nvalid = min(32, p.rows_b - col0);
                    if (row_ok && nvalid > 0) {
                        float v[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            v[j] = __uint_as_float(r[j]);
                            if constexpr (EPI == kPairRelu2) {
                                v[j] = fmaxf(Cvt<T>::to_f(Cvt<T>::from_f(v[j])), 0.f);
                                v[j] *= v[j];
                            }
                        }
                        epilogue_store<T>(p, v, row, col0, nvalid);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(&tempty_bar[acc], 0);
        }
    }

    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_w();       // the other CTA's tensor core may still be reading this CTA's tiles / TMEM
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc2(tmem_base, 512);
    }
}

template <typename T, int EPI>
static int launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t stream) {
    auto kern = gemm_pair_kernel<T, EPI>;
    static const int max_pairs = resident_pairs(kern, kPairThreads, kPairSmem);
    if (max_pairs <= 0) return fail("gemm_pair: configuration");
    const int total = p.tiles_a * p.tiles_b;
    const cudaError_t e = launch_pairs(kern, total < max_pairs ? total : max_pairs, kPairThreads, kPairSmem, stream, ta, tb, p);
    if (e != cudaSuccess) return fail("cudaLaunchKernelEx(gemm_pair)", e);
    return 0;
}

}  // namespace telb

using namespace telb;

// Whether M x N outputs take the pair kernel.  Both kernels work in whole waves of tiles (74 pairs of 256 x 256, 148 CTAs of 128 x 256);
// a pair's wave takes 0.82 of the single CTA's (8129 x 24576 x 4096: 42 waves, 1035 against 1270 us), so it pays unless the larger tile
// needs that many more waves: 1030 x 24576 x 4096: 7 against 6 waves, 203 against 216 us; 1030 x 4096 x 12288: 2 against 1, 173 against 102 us.
extern "C" int telb_gemm_skinny_pays(int M, int N, int K);
extern "C" int telb_gemm_pair_pays(int M, int N, int K) {
    if (M <= 128 || N < 256 || telb_gemm_skinny_pays(M, N, K)) return 0;
    const long long sms = sm_count(), nb = (N + 255) / 256;
    const long long pair = ((M + 255) / 256 * nb + sms / 2 - 1) / (sms / 2), single = ((M + 127) / 128 * nb + sms - 1) / sms;
    return pair * 82 < single * 100;
}

// epi: 0 plain (bias, alpha, residual may be null), 1 SwiGLU over w [2 N, K] (gate rows first), 2 squared ReLU; 1 and 2 take no bias, scale
// or residual.  K % 8 == 0, operands 16-byte aligned.
extern "C" int telb_gemm_pair(const void* x, const void* w, void* out, int M, int N, int K, const void* bias, const float* alpha,
                              const void* residual, int epi, int is_bf16, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (K % 8) return fail("telb_gemm_pair: K must be a multiple of 8");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return fail("telb_gemm_pair: operands must be 16-byte aligned");
    if (epi != kPairPlain && (bias || alpha || residual)) return fail("telb_gemm_pair: the activation forms take no bias, scale or residual");
    const CUtensorMapDataType dt = is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    GemmParams p{};
    p.k = K;
    p.kb_total = (K + kBK - 1) / kBK;
    p.kb_per_split = p.kb_total;
    p.splits = 1;
    p.c = out;
    p.bias = bias;
    p.alpha = alpha;
    p.residual = residual;
    p.out_bf16 = is_bf16;
    p.status = status;
    p.rows_a = M;
    p.rows_b = N;
    p.ldc_lane = N;
    p.ldc_col = 1;
    p.tiles_a = (M + 255) / 256;
    p.tiles_b = epi == kPairSwiglu ? (N + 127) / 128 : (N + kPairBN - 1) / kPairBN;
    CUtensorMap ta, tb;
    if (make_tmap_2d(&ta, dt, 2, x, M, K, (uint64_t)K * 2, 128, kBK, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (make_tmap_2d(&tb, dt, 2, w, (uint64_t)N * (epi == kPairSwiglu ? 2 : 1), K, (uint64_t)K * 2, 128, kBK, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
#define TELB_PAIR(T_) (epi == kPairSwiglu ? launch_gemm_pair<T_, kPairSwiglu>(ta, tb, p, stream) : epi == kPairRelu2 ? launch_gemm_pair<T_, kPairRelu2>(ta, tb, p, stream) : launch_gemm_pair<T_, kPairPlain>(ta, tb, p, stream))
    return is_bf16 ? TELB_PAIR(__nv_bfloat16) : TELB_PAIR(__half);
#undef TELB_PAIR
}
