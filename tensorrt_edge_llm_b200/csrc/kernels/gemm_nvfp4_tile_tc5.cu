// NVFP4 block-scaled GEMM for prefill-size M, 128 x 256 output tiles, one persistent CTA per SM:
//     out[M,N] = (xq ⊙ sfx)[M,K] · (wq ⊙ sfw)[N,K]ᵀ · alpha[N]  (+ bias, + residual)
//
// What bounds it: a K step of 256 is 16.8 MFLOP (0.27 us at the fp4 rate) and 54 KB from L2.  Loads alone stream at 22 TB/s, which
// is 6.8 PFLOP/s at 8192 x 24576 x 4096 (242 us); everything else has to hide behind them.  Two things did not:
//   * Scale factors.  Twelve `tcgen05.cp` per K step in front of the four MMAs run in the tensor pipe's order and cost as much as 40
//     cycles each (479 us without stores, 304 us with the copies left out).  Here a warp per TMEM lane quadrant carries them through
//     registers instead (`tcgen05.st` of 48 columns), one K step ahead of the MMAs: 354 us.
//   * The epilogue.  Two 256-column accumulators do not fit beside the scale columns, so they overlap by 128 columns and the next
//     tile's MMAs wait for half of this one.  Eight epilogue warps take that half into registers with two loads each and release it
//     before they scale, convert and store anything.
//
// TMEM plan (512 columns): [0,256) accumulator 0, [128,384) accumulator 1, [384,480) two scale buffers of 48 columns.
// Roles (14 warps): 0 TMA producer, 1 MMA issuer / TMEM owner, 2-9 epilogue (two warps per lane quadrant, 64 columns of a half each),
// 10-13 scale factors.  Every wait is bounded.
//
// Grouped form (mixture of experts): a row tile belongs to one expert, `tile_expert` names its weight block and how many of its rows are in
// use.  Tiles of few rows (a decode step routes two or three tokens to an expert) load 32 rows of x instead of 128.  Their K loops are
// short (3 to 8 steps), so the column scales are fetched to shared memory while the MMAs run.
//
// RS: the reduce-scatter form stages rows in shared memory so that they leave as 128-byte lines to their owner rank, in the place of
// the fourth operand stage.  No TMA load here uses cluster multicast (the kernel runs inside tensor-parallel steps too).
#include "gemm_common.cuh"
#include "nvfp4_common.cuh"

namespace telb {

constexpr int kNtBN = 256;
constexpr int kNtAcc1 = 128;                // first column of accumulator 1
constexpr int kNtSf0 = 384;                 // first scale-factor column
constexpr int kNtSfCols = 48;               // 16 of the rows, 32 of the weights
constexpr int kNtEpiWarps = 8;
constexpr int kNtThreads = 32 * (2 + kNtEpiWarps + 4);

template <bool RS>
struct NtCfg {
    static constexpr int kATile = 128 * 128;
    static constexpr int kBTile = 256 * 128;
    static constexpr int kSf = 2048 + 4096;
    static constexpr int kStage = kATile + kBTile + kSf;
    static constexpr int kStages = RS ? 3 : 4;
    static constexpr int kSlab = RS ? kNtEpiWarps * 32 * kRsStageRowBytes : 0;
    static constexpr int kSmem = kStages * kStage + 1024 + 256 + kSlab + (RS ? 0 : kNtEpiWarps * 128 * 4);
};

struct NtTile {
    int a0, b0, tb;
    int brow;              // first weight row of the tile's expert (0: one weight for all rows)
    int rows;              // rows of the tile in use; 0 = nothing to do
};
__device__ __forceinline__ NtTile nt_tile(const GemmParams& p, int t) {
    const int per_group = kRasterGroup * p.tiles_b;
    const int group = t / per_group;
    const int within = t - group * per_group;
    const int gfirst = group * kRasterGroup;
    const int gsize = min(kRasterGroup, p.tiles_a - gfirst);
    NtTile w;
    w.a0 = (gfirst + within % gsize) * kBM;
    w.tb = within / gsize;
    w.b0 = w.tb * kNtBN;
    w.brow = 0;
    w.rows = 128;
    if (p.tile_expert) {
        const int ta = w.a0 / kBM, e = p.tile_expert[ta];
        w.rows = e < 0 ? 0 : p.tile_expert[p.tiles_a + ta];
        w.brow = max(e, 0) * p.group_rows_b;
    }
    return w;
}

__device__ __forceinline__ void st_global_32b(void* dst, const uint4& a, const uint4& b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(dst), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}

// 32 gate and 32 up sums of one row → 32 quantised SwiGLU outputs (features f0 .. f0 + 31): the same roundings as the unfused
// chain (16-bit GEMM output, 16-bit activation), then quantise.
template <typename T>
__device__ __forceinline__ void nt_swiglu(const GemmParams& p, const uint32_t (&rg)[32], const uint32_t (&ru)[32], int row, const float* ga, const float* ua, int f0,
                                          float gs, float inv_gs) {
    uint2 packed[2];
    uint8_t s8[2];
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
        float y[16];
        float amax = 0.f;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int j = hf * 16 + k;
            float g = __uint_as_float(rg[j]), u = __uint_as_float(ru[j]);
            if (ga) {
                g *= ga[j];
                u *= ua[j];
            }
            g = Cvt<T>::to_f(Cvt<T>::from_f(g));
            u = Cvt<T>::to_f(Cvt<T>::from_f(u));
            y[k] = Cvt<T>::to_f(Cvt<T>::from_f(g / (1.f + __expf(-g)) * u));
            amax = fmaxf(amax, fabsf(y[k]));
        }
        packed[hf] = nvfp4_quantize_block16(y, amax, gs, inv_gs, s8[hf]);
    }
    // f0 is a multiple of 32: 16 bytes of codes, and two scales that share a half word of their atom
    uint8_t* dst = p.sw_xq + (size_t)row * p.sw_ld + (f0 >> 1);
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0].x, packed[0].y, packed[1].x, packed[1].y);
    } else {
        *reinterpret_cast<uint2*>(dst) = packed[0];
        *reinterpret_cast<uint2*>(dst + 8) = packed[1];
    }
    uint8_t* sf = p.sw_sf + sf_atom_offset((long long)row, f0 >> 4, p.sw_k64_pad);
    *reinterpret_cast<uint16_t*>(sf) = static_cast<uint16_t>(s8[0] | (s8[1] << 8));
}

// 32 columns of one row.  Whole 32-byte sectors leave with one store each where the row pitch allows it.
template <typename T>
__device__ __forceinline__ void nt_store32(const GemmParams& p, const uint32_t (&r)[32], int row, int col0, bool wide_rows) {
    const int nvalid = min(32, p.rows_b - col0);
    if (nvalid <= 0) return;
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
    if (wide_rows && nvalid == 32) {
        uint4 u[4];
        pack_chunk<T>(p, v, col0, u);
        T* dst = reinterpret_cast<T*>(p.c) + (size_t)row * p.ldc_lane + col0;
        st_global_32b(dst, u[0], u[1]);
        st_global_32b(dst + 16, u[2], u[3]);
    } else {
        epilogue_store<T>(p, v, row, col0, nvalid);
    }
}

template <bool RS>
__global__ void __launch_bounds__(kNtThreads, 1)
gemm_nvfp4_tile_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_a32,
                       const __grid_constant__ CUtensorMap tma_b, const uint8_t* __restrict__ sf_a,
                       const uint8_t* __restrict__ sf_b, int sf_k64, GemmParams p) {
    using Cfg = NtCfg<RS>;
    constexpr int STAGES = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::kStage);
    uint64_t* sfull_bar = full_bar + STAGES;           // a stage's scale factors are in shared memory
    uint64_t* empty_bar = sfull_bar + STAGES;
    uint64_t* tsf_bar = empty_bar + STAGES;            // a scale buffer in TMEM is filled
    uint64_t* tsfe_bar = tsf_bar + 2;                  // ... has been read by its MMAs
    uint64_t* tfull_bar = tsfe_bar + 2;
    uint64_t* tempty_bar = tfull_bar + 2;
    uint64_t* tovl_bar = tempty_bar + 2;               // the half that the next accumulator overlaps is drained
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tovl_bar + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    uint8_t* slab0 = smem + STAGES * Cfg::kStage + 256;
    float* s_alpha = reinterpret_cast<float*>(slab0);      // column scales of the tile, 128 per epilogue warp (grouped form, which has no slab)

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int total_tiles = p.tiles_a * p.tiles_b;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&sfull_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tsf_bar[s], 4);
            mbar_init(&tsfe_bar[s], 1);
            mbar_init(&tfull_bar[s], 1);
            mbar_init(&tempty_bar[s], kNtEpiWarps);
            mbar_init(&tovl_bar[s], kNtEpiWarps);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tensormap(&tma_a);
        prefetch_tensormap(&tma_b);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    pdl_prologue();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- producer ----------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            const int ag_e = p.ag_flags ? *p.ag_epoch : 0;
            const int last_a = (p.rows_a - 1) / 128, last_b = (p.rows_b - 1) / 128;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                const NtTile w = nt_tile(p, t);
                if (w.rows == 0) continue;
                const bool few = w.rows <= 32;
                const int eb = w.brow / 128;
                if (p.ag_flags && !ag_wait_rows(p, w.a0, ag_e, abort_flag)) break;
                const uint8_t* ga = sf_a + (size_t)min(w.a0 / 128, last_a) * sf_k64 * 512;
                const uint8_t* gb0 = sf_b + (size_t)(eb + min(w.b0 / 128, last_b)) * sf_k64 * 512;
                const uint8_t* gb1 = sf_b + (size_t)(eb + min(w.b0 / 128 + 1, last_b)) * sf_k64 * 512;
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kStatusProducerTimeout)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sa = smem + stage * Cfg::kStage;
                    uint8_t* sb = sa + Cfg::kATile;
                    uint8_t* ss = sb + Cfg::kBTile;
                    mbar_expect_tx(&sfull_bar[stage], Cfg::kSf);
                    bulk_load(ss, ga + (size_t)kb * 2048, 2048, &sfull_bar[stage]);
                    bulk_load(ss + 2048, gb0 + (size_t)kb * 2048, 2048, &sfull_bar[stage]);
                    bulk_load(ss + 4096, gb1 + (size_t)kb * 2048, 2048, &sfull_bar[stage]);
                    mbar_expect_tx(&full_bar[stage], (few ? Cfg::kATile / 4 : Cfg::kATile) + Cfg::kBTile);
                    tma_load_2d(sa, few ? &tma_a32 : &tma_a, &full_bar[stage], kb * 128, w.a0);      // few: the other rows keep what was there
                    tma_load_2d(sb, &tma_b, &full_bar[stage], kb * 128, w.brow + w.b0);
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            const uint32_t idesc = idesc_nvfp4(128, kNtBN);
            int stage = 0;
            uint32_t phase = 0, buf = 0, bphase = 0;
            bool ok = true;
            int i = -1;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                if (nt_tile(p, t).rows == 0) continue;
                ++i;
                const int acc = i & 1;
                const uint32_t use_par = (uint32_t)(i >> 1) & 1u;
                // the accumulator's previous tile is fully drained, and the previous tile's overlapping half is drained
                if (!mbar_wait(&tempty_bar[acc], use_par ^ 1, abort_flag, p.status, kStatusMmaTimeout)) break;
                if (i > 0 && !mbar_wait(&tovl_bar[acc ^ 1], (uint32_t)((i - 1) >> 1) & 1u, abort_flag, p.status, kStatusMmaTimeout)) break;
                const uint32_t d_tmem = tmem_base + (acc ? kNtAcc1 : 0);
                for (int kb = 0; kb < p.kb_total; ++kb) {
                    if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, kStatusMmaTimeout) ||
                        !mbar_wait(&tsf_bar[buf], bphase, abort_flag, p.status, kStatusMmaTimeout)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint8_t* sa = smem + stage * Cfg::kStage;
                    const uint32_t t_sfa = tmem_base + kNtSf0 + buf * kNtSfCols;
                    const uint64_t da = smem_desc_sw128(sa);
                    const uint64_t db = smem_desc_sw128(sa + Cfg::kATile);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        umma_nvfp4(d_tmem, da + 2 * q, db + 2 * q, idesc, t_sfa + q * 4, t_sfa + 16 + q * 8, (kb > 0 || q > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[stage]);
                    umma_commit(&tsfe_bar[buf]);
                    bphase ^= buf;
                    buf ^= 1;
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit(&tfull_bar[acc]);
            }
        }
    } else if (warp >= 2 + kNtEpiWarps) {
        // ---------------- scale factors: 32 rows x 16 bytes of an atom, the same in every lane quadrant ----------------
        int stage = 0;
        uint32_t phase = 0, buf = 0, bphase = 0;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + kNtSf0;
        bool ok = true;
        for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
            if (nt_tile(p, t).rows == 0) continue;
            for (int kb = 0; kb < p.kb_total; ++kb) {
                if (!mbar_wait(&sfull_bar[stage], phase, abort_flag, p.status, kStatusMmaTimeout)) {
                    ok = false;
                    break;
                }
                const uint8_t* ss = smem + stage * Cfg::kStage + Cfg::kATile + Cfg::kBTile + lane * 16;
                uint32_t ra[16], rb[32];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 a = *reinterpret_cast<const uint4*>(ss + q * 512);
                    const uint4 b0 = *reinterpret_cast<const uint4*>(ss + 2048 + q * 512);
                    const uint4 b1 = *reinterpret_cast<const uint4*>(ss + 4096 + q * 512);
                    ra[q * 4] = a.x, ra[q * 4 + 1] = a.y, ra[q * 4 + 2] = a.z, ra[q * 4 + 3] = a.w;
                    rb[q * 8] = b0.x, rb[q * 8 + 1] = b0.y, rb[q * 8 + 2] = b0.z, rb[q * 8 + 3] = b0.w;
                    rb[q * 8 + 4] = b1.x, rb[q * 8 + 5] = b1.y, rb[q * 8 + 6] = b1.z, rb[q * 8 + 7] = b1.w;
                }
                if (!mbar_wait(&tsfe_bar[buf], bphase ^ 1, abort_flag, p.status, kStatusMmaTimeout)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                tmem_st_x16(lane_addr + buf * kNtSfCols, ra);
                tmem_st_x32(lane_addr + buf * kNtSfCols + 16, rb);
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&tsf_bar[buf]);
                bphase ^= buf;
                buf ^= 1;
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    } else {
        // ---------------- epilogue: lane quadrant `quad`, column group `grp` of every half ----------------
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        const bool wide_rows = !p.residual && p.rows_b % 16 == 0 && (reinterpret_cast<uintptr_t>(p.c) & 31) == 0;
        int i = -1;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
            const NtTile w = nt_tile(p, t);
            if (w.rows == 0) continue;
            ++i;
            const int acc = i & 1;
            const bool sw = p.sw_xq != nullptr;
            // SwiGLU: columns [0,64) of a half are gate features, [64,128) the matching up features; 32 of each per warp
            const int c0 = sw ? grp * 32 : grp * 64, c1 = sw ? 64 + grp * 32 : grp * 64 + 32;
            const float* buf = nullptr;
            if (!RS && p.tile_expert && p.alpha) {
                float* own = s_alpha + (warp - 2) * 128;
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int col = w.b0 + (q >> 1) * 128 + ((q & 1) ? c1 : c0) + lane;
                    own[q * 32 + lane] = col < p.rows_b ? __ldg(&p.alpha[w.brow + col]) : 0.f;
                }
                __syncwarp();
                buf = own;
            }
            if (!mbar_wait(&tfull_bar[acc], (uint32_t)(i >> 1) & 1u, abort_flag, p.status, kStatusEpilogueTimeout)) break;
            tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + (acc ? kNtAcc1 : 0);
            const int row = w.a0 + quad * 32 + lane;
            const bool row_ok = row < p.rows_a && quad * 32 + lane < w.rows;
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
                // accumulator 0 gives up its upper half first (accumulator 1 begins there), accumulator 1 its lower half
                const int h = acc ? hh : (hh ^ 1);
                const int hb0 = w.b0 + h * 128;
                // scales of the two 32-column pieces of this half
                const float* a0 = buf ? buf + h * 64 : p.alpha ? p.alpha + hb0 + c0 : nullptr;
                const float* a1 = buf ? buf + h * 64 + 32 : p.alpha ? p.alpha + hb0 + c1 : nullptr;
                uint32_t r0[32], r1[32];
                tmem_ld_x32(t_addr + h * 128 + c0, r0);
                tmem_ld_x32(t_addr + h * 128 + c1, r1);
                tmem_ld_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(hh == 0 ? &tovl_bar[acc] : &tempty_bar[acc]);
                if (sw) {
                    if (row_ok && hb0 + 128 <= p.rows_b) {
                        const float gs = *p.sw_gs;
                        const int f0 = (w.tb * 2 + h) * 64 + grp * 32;
                        if (p.out_bf16) nt_swiglu<__nv_bfloat16>(p, r0, r1, row, a0, a1, f0, gs, 1.f / gs);
                        else nt_swiglu<__half>(p, r0, r1, row, a0, a1, f0, gs, 1.f / gs);
                    }
                } else if (RS) {
                    uint8_t* slab = slab0 + (warp - 2) * (32 * kRsStageRowBytes);
                    const int seg = lane & 7, rsub = lane >> 3;
                    float v[32];
                    uint4 u[4];
#pragma unroll
                    for (int s2 = 0; s2 < 2; ++s2) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(s2 ? r1[j] : r0[j]);
                        const int col0 = min(hb0 + c0 + s2 * 32, max(p.rows_b - 32, 0));   // clamp: columns past N are not stored
                        if (p.out_bf16) pack_chunk<__nv_bfloat16>(p, v, col0, u);
                        else pack_chunk<__half>(p, v, col0, u);
                        uint4* dst = reinterpret_cast<uint4*>(slab + lane * kRsStageRowBytes + s2 * 64);
#pragma unroll
                        for (int q = 0; q < 4; ++q) dst[q] = u[q];
                    }
                    __syncwarp();
                    const int colseg = hb0 + c0 + seg * 8;
#pragma unroll
                    for (int rr = 0; rr < 32; rr += 4) {
                        const int lr = rr + rsub;
                        const int grow = w.a0 + quad * 32 + lr;
                        if (grow < p.rows_a && colseg + 8 <= p.rows_b) {
                            const int d = grow / p.rs_rows_per_rank;
                            const size_t orow = (size_t)p.rs_rank * p.rs_rows_per_rank + (grow - d * p.rs_rows_per_rank);
                            const uint4 val = *reinterpret_cast<const uint4*>(slab + lr * kRsStageRowBytes + seg * 16);
                            uint16_t* base = reinterpret_cast<uint16_t*>(p.rs_out[d]);
                            *reinterpret_cast<uint4*>(base + orow * (size_t)p.ldc_lane + colseg) = val;
                        }
                    }
                    __syncwarp();
                } else if (row_ok) {
                    GemmParams p0 = p, p1 = p;
                    if (buf) {
                        p0.alpha = a0 - (hb0 + c0);
                        p1.alpha = a1 - (hb0 + c1);
                    }
                    if (p.out_bf16) {
                        nt_store32<__nv_bfloat16>(p0, r0, row, hb0 + c0, wide_rows);
                        nt_store32<__nv_bfloat16>(p1, r1, row, hb0 + c1, wide_rows);
                    } else {
                        nt_store32<__half>(p0, r0, row, hb0 + c0, wide_rows);
                        nt_store32<__half>(p1, r1, row, hb0 + c1, wide_rows);
                    }
                }
            }
        }
        // the peer stores of the reduce-scatter epilogue are performed system-wide before the kernel ends, so the
        // "GEMM finished" flag the next kernel publishes can never overtake them
        if (RS) __threadfence_system();
    }

    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

template <bool RS>
static int launch_tile(const CUtensorMap& ta, const CUtensorMap& ta32, const CUtensorMap& tb, const uint8_t* sfa, const uint8_t* sfb, int k64, const GemmParams& p,
                       cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_nvfp4_tile_kernel<RS>, cudaFuncAttributeMaxDynamicSharedMemorySize, NtCfg<RS>::kSmem);
        if (e != cudaSuccess) return fail("cudaFuncSetAttribute(gemm_nvfp4_tile)", e);
        configured = true;
    }
    const int total = p.tiles_a * p.tiles_b;
    const int grid = total < sm_count() ? total : sm_count();
    TELB_LAUNCH("gemm_nvfp4_tile_kernel", (gemm_nvfp4_tile_kernel<RS>), dim3(grid), dim3(kNtThreads), NtCfg<RS>::kSmem, stream, ta, ta32, tb, sfa, sfb, k64, p);
    TELB_CHECK_LAUNCH("gemm_nvfp4_tile_kernel");
    return 0;
}

}  // namespace telb

using namespace telb;

// Large-M layout (M > 128 is the caller's business; any M works).  `params_blob`: a GemmParams with the epilogue / fusion fields set;
// this fills the tile geometry and launches.
extern "C" int telb_gemm_nvfp4_tile_launch(const void* xq, const void* x_sf, const void* wq, const void* w_sf, int M, int N, int K,
                                           const void* params_blob, cudaStream_t stream) {
    GemmParams p = *static_cast<const GemmParams*>(params_blob);
    if (K % 32) return fail("telb_gemm_nvfp4_tile: K must be a multiple of 32");
    if (N % 8) return fail("telb_gemm_nvfp4_tile: N must be a multiple of 8");
    const uint64_t kbytes = (uint64_t)K / 2;
    p.k = K;
    p.kb_total = (K + 255) / 256;
    p.rows_a = M;
    p.rows_b = N;
    p.ldc_lane = N;
    p.ldc_col = 1;
    p.feat_on_lane = 0;
    p.splits = 1;
    p.kb_per_split = p.kb_total;
    p.tiles_a = (M + kBM - 1) / kBM;
    p.tiles_b = (N + kNtBN - 1) / kNtBN;
    CUtensorMap ta, tb;
    if (make_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, M, kbytes, kbytes, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (make_tmap_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, N, kbytes, kbytes, 256, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    const int k64 = p.kb_total * 4;
    return p.rs_world > 1 ? launch_tile<true>(ta, ta, tb, (const uint8_t*)x_sf, (const uint8_t*)w_sf, k64, p, stream)
                          : launch_tile<false>(ta, ta, tb, (const uint8_t*)x_sf, (const uint8_t*)w_sf, k64, p, stream);
}

// Grouped form: `params_blob` carries the epilogue fields, tile_expert and the weight rows per expert (rows_b = group_rows_b = N).
extern "C" int telb_gemm_nvfp4_tile_grouped_launch(const void* xq, const void* x_sf, const void* wq, const void* w_sf, int rows_pad, int K, int experts,
                                                   const void* params_blob, cudaStream_t stream) {
    GemmParams p = *static_cast<const GemmParams*>(params_blob);
    const uint64_t kbytes = (uint64_t)K / 2;
    p.kb_total = (K + 255) / 256;
    p.tiles_a = rows_pad / kBM;
    p.tiles_b = (p.rows_b + kNtBN - 1) / kNtBN;
    CUtensorMap ta, ta32, tb;
    if (make_tmap_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, rows_pad, kbytes, kbytes, 128, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (make_tmap_2d(&ta32, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, rows_pad, kbytes, kbytes, 32, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (make_tmap_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, (uint64_t)experts * p.rows_b, kbytes, kbytes, 256, 128, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    return launch_tile<false>(ta, ta32, tb, (const uint8_t*)x_sf, (const uint8_t*)w_sf, p.kb_total * 4, p, stream);
}
