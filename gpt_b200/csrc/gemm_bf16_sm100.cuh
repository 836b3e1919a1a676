// Products of more than a few rows with a bf16 weight matrix stored [n][k]: out[m][n] = a[m][k] . w[n][k], fp32 accumulation, every OutKind.
//
// A CTA pair (cta_group::2) computes tiles of 256 x BN: each CTA loads its own 128 rows of A and half of the BN rows of w, 64 values of k (128-byte rows,
// 128-byte swizzle) per stage; one thread of the leader issues 256 x BN x 16 instructions into one of two accumulators in TMEM.  Whole tiles, as evenly as
// they go, m fastest (the pairs that run together share rows of w in L2).
//
// What bounds it: the tensor pipe and the power limit at large sizes (4096 x 10304 x 2048: 1 530 TFLOP/s, 113 us; loads alone 57 us, instructions alone
// 86 us), the last wave and the first loads at small ones.  The general pair kernel (gemm_sm100_pair.cuh) took 167 us: it built two 64-bit descriptors per
// instruction in the issuing thread, waited with cluster-scope acquires, and cut tiles between pairs, which costs more than it saves while a tile's main
// loop is a few microseconds (2611 x 3072 x 768: 33 us against 15 us).
//
// The accumulator adds with truncation, so a sum of many instructions loses more than fp32 additions would: after kBf16Chunk k-blocks the accumulator goes
// to running sums in the epilogue's registers (round to nearest) while the other one is filled.
#pragma once

#include "gemm_sm100.cuh"

namespace gptb200 {

struct Bf16GemmParams {
    int M, N, num_kb;       // k-blocks of 64
    int tiles_m, tiles_n;   // tiles of 256 rows and of BN columns
    int *status;
    const float *bias;      // null: none
    int glu;                // gated kinds: OUT_GLU or OUT_GLU_SILU
    float *tail;            // OUT_BF16, as in GemmParams
    int tail_col, tail_pitch;
    int silu_cols;
    const uint16_t *factor; // OUT_GELU_MUL
    const int *factor_rows;
    int factor_pitch;
    int a_group_cols, a_group_rows;
};

constexpr int kBf16Chunk = 16;   // k-blocks per hand-off of the accumulator: 64 instructions

enum Bf16Form : int { BF16_F32 = 0, BF16_PLAIN = 1, BF16_GLU = 2, BF16_FACTOR = 3 };

template <int BN>
struct Bf16Cfg {
    static constexpr int kStages = BN == 256 ? 6 : BN == 128 ? 8 : 9;
    static constexpr int kBBytes = BN / 2 * 128;
    static constexpr int kStageBytes = kATileBytes + kBBytes;
    static constexpr int kEpiWarps = 8;               // two per TMEM lane quarter, BN / 2 columns each
    static constexpr int kCols = BN / 2;
    static constexpr int kPiece = kCols < 64 ? kCols : 64;   // columns of a 16-bit piece before packing: rows of 128 bytes where a warp has enough
    static constexpr int kStagingBytes = kEpiWarps * 4096;
    static constexpr int kThreads = (4 + kEpiWarps) * 32;
    static constexpr int kBarriers = 2 * kStages + 5;
    static constexpr int kSmemBytes = kStages * kStageBytes + kStagingBytes + 1024 + 256;
    static_assert(8 * kBarriers + 8 <= 256 && kSmemBytes <= 232448, "shared memory");
};

// Words per row of an output box: a piece as it is stored.
__host__ __device__ constexpr int bf16_out_box(int bn, int form) { return form == BF16_F32 ? 32 : form == BF16_GLU || bn == 64 ? 16 : 32; }

template <int BN, int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Bf16Cfg<BN>::kThreads, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_out,
                      const Bf16GemmParams p)
{
    using C = Bf16Cfg<BN>;
    static_assert(FORM != BF16_GLU || C::kCols >= 64, "a gate and its up column belong to one warp");
    constexpr int STAGES = C::kStages;
    constexpr int kTmemCols = 2 * BN;
    constexpr uint32_t kIdesc = ptx::make_idesc_bf16(256, BN, false, false);

    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    const uint32_t staging_base = smem_base + STAGES * C::kStageBytes;
    const uint32_t bar_base = staging_base + C::kStagingBytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };                   // used in the leader: the loads of both CTAs
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
    auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };   // used in the leader
    const uint32_t drain_bar = bar_base + 8u * (2 * STAGES + 4);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + (bar_base - smem_base) + 8 * C::kBarriers);
    volatile uint32_t *abort_flag = tmem_slot + 1;

    const int warp = ptx::warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();
    const bool leader = rank == 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(full_bar(s), 1);
            ptx::mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(tmem_full_bar(b), 1);
            ptx::mbar_init(tmem_empty_bar(b), 2 * C::kEpiWarps);
        }
        ptx::mbar_init(drain_bar, 1);
        *abort_flag = 0u;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_a);
        ptx::prefetch_tensormap(&tmap_w);
        ptx::prefetch_tensormap(&tmap_out);
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(ptx::smem_u32(tmem_slot), kTmemCols);
        ptx::tmem_relinquish_pair();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();   // the peer's barriers exist before anything is signalled across CTAs
    ptx::tc_fence_after();
    const uint32_t tmem_base = ptx::warp_uniform(*tmem_slot);
    grid_dependency_wait();      // the set-up above overlaps the predecessor's last CTAs
    if (threadIdx.x == 0) grid_dependency_launch();

    const int pairs = gridDim.x >> 1, pair = blockIdx.x >> 1, tiles = p.tiles_m * p.tiles_n;

    if (warp < 4) {
        ptx::reg_dec<72>();
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer (both CTAs): the warp walks, one lane issues
            const bool issuer = ptx::elect_one();
            uint32_t s = 0, ph = 0;
            bool ok = true;
            for (int t = pair; ok && t < tiles; t += pairs) {
                const int tn = t / p.tiles_m, tm = t - tn * p.tiles_m;
                const int m0 = tm * 256 + static_cast<int>(rank) * 128 + (p.a_group_cols ? tn * BN / p.a_group_cols * p.a_group_rows : 0);
                const int n0 = tn * BN + static_cast<int>(rank) * (BN / 2);
                for (int kb = 0; kb < p.num_kb; ++kb) {
                    if (!bounded_wait(empty_bar(s), ph ^ 1u, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) {
                        ok = false;
                        break;
                    }
                    if (issuer) {
                        const uint32_t bar = ptx::map_to_cta(full_bar(s), 0u), dst = smem_base + s * C::kStageBytes;
                        if (leader) ptx::mbar_arrive_expect_tx(full_bar(s), 2 * C::kStageBytes);
                        ptx::tma_load_2d_pair(dst, &tmap_a, kb * kBK, m0, bar);
                        ptx::tma_load_2d_pair(dst + kATileBytes, &tmap_w, kb * kBK, n0, bar);
                    }
                    __syncwarp();
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        } else if (warp == 1 && leader) {
            // ------------------------------------------------------------ MMA issuer (leader CTA): the warp walks, one lane issues
            const bool issuer = ptx::elect_one();
            uint32_t s = 0, ph = 0, g = 0;
            bool ok = true;
            const ptx::SmemDesc desc_a = ptx::smem_desc_words(smem_base, 16, 1024, ptx::kLayoutSw128);
            const ptx::SmemDesc desc_w = ptx::smem_desc_words(smem_base + kATileBytes, 16, 1024, ptx::kLayoutSw128);
            for (int t = pair; ok && t < tiles; t += pairs) {
                for (int kb = 0; ok && kb < p.num_kb; ++g) {
                    const int kend = min(kb + kBf16Chunk, p.num_kb);
                    const uint32_t buf = g & 1u, use = (g >> 1) & 1u;
                    if (!bounded_wait(tmem_empty_bar(buf), use ^ 1u, abort_flag, p.status, DEV_TIMEOUT_MMA_TMEM)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * BN;
                    uint32_t accumulate = 0;
                    for (; kb < kend; ++kb) {
                        if (!bounded_wait(full_bar(s), ph, abort_flag, p.status, DEV_TIMEOUT_MMA_FULL)) {
                            ok = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        const uint32_t at = s * C::kStageBytes;
                        if (issuer) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) ptx::mma_f16_ss_pair(d_tmem, desc_a.at(at + k * 32), desc_w.at(at + k * 32), kIdesc, k ? 1u : accumulate);
                            ptx::mma_commit_pair_both(empty_bar(s), 3);   // the stage is free in both CTAs once these have read it
                        }
                        accumulate = 1u;
                        if (++s == STAGES) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    if (ok && issuer) ptx::mma_commit_pair_both(tmem_full_bar(buf), 3);
                }
            }
            if (issuer) ptx::mma_commit_pair(drain_bar);   // do not leave with instructions still running: they write TMEM that is about to be released
            bounded_wait(drain_bar, 0u, abort_flag, p.status, DEV_TIMEOUT_DRAIN);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
        ptx::reg_inc<216>();   // 128 x 72 + 256 x 216 = 384 x 168 registers
        const int e = warp - 4, q = warp & 3, col_base = (e >> 2) * C::kCols;
        const uint32_t tmem_mine = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + col_base;
        const uint32_t stage = staging_base + e * 4096;
        const uint32_t leader_empty[2] = {ptx::map_to_cta(tmem_empty_bar(0), 0u), ptx::map_to_cta(tmem_empty_bar(1), 0u)};
        uint32_t g = 0;
        bool ok = true;
        // One staged box goes out: the warp's rows x `box` words, first word `word`.
        auto send = [&](int word, int row0, bool inside) {
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                if (inside) ptx::tma_store_3d(&tmap_out, word, row0, 0, stage);
                ptx::tma_store_commit();
            }
        };
        auto staging_free = [&]() {
            if (lane == 0) ptx::tma_store_wait_read<0>();
            __syncwarp();
        };
        for (int t = pair; ok && t < tiles; t += pairs) {
            const int tn = t / p.tiles_m, tm = t - tn * p.tiles_m;
            const int row0 = tm * 256 + static_cast<int>(rank) * 128 + q * 32, n0 = tn * BN + col_base;
            float acc[C::kCols];
#pragma unroll
            for (int j = 0; j < C::kCols; ++j) acc[j] = 0.0f;
            for (int kb = 0; kb < p.num_kb; kb += kBf16Chunk, ++g) {
                const uint32_t buf = g & 1u, use = (g >> 1) & 1u;
                if (!bounded_wait(tmem_full_bar(buf), use, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
#pragma unroll
                for (int c = 0; c < C::kCols; c += 32) {
                    uint32_t v[32];
                    ptx::tmem_ld_32x32(tmem_mine + buf * BN + c, v);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[c + j] += __uint_as_float(v[j]);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive_remote(leader_empty[buf]);
            }
            if (!ok) break;
            if (p.bias) {
#pragma unroll
                for (int c = 0; c < C::kCols; c += 32) {
                    const float b = n0 + c + lane < p.N ? __ldg(p.bias + n0 + c + lane) : 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[c + j] += __shfl_sync(0xffffffffu, b, j);
                }
            }
            const bool rows_inside = row0 < p.M, mine = row0 + lane < p.M;
            // One copy of the code for all pieces, the sums move down: straight-line code for all of them comes through the instruction caches once per launch
            // and costs more than the moves.
#pragma unroll 1
            for (int c = 0; c < C::kCols; c += C::kPiece) {
                const int col = n0 + c;
                if constexpr (FORM == BF16_F32) {
#pragma unroll
                    for (int h = 0; h < C::kPiece; h += 32) {
                        staging_free();
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            ptx::sts128(stage + lane * 128 + ((j ^ (lane & 7)) << 4), __float_as_uint(acc[h + 4 * j]), __float_as_uint(acc[h + 4 * j + 1]),
                                        __float_as_uint(acc[h + 4 * j + 2]), __float_as_uint(acc[h + 4 * j + 3]));
                        send(col + h, row0, rows_inside && col + h < p.N);
                    }
                } else if constexpr (FORM == BF16_GLU) {
                    uint32_t w[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float a = acc[2 * j], b = acc[2 * j + 1];
                        const float ga = p.glu == OUT_GLU ? gelu_tanh(a) : silu_fast(a), gb = p.glu == OUT_GLU ? gelu_tanh(b) : silu_fast(b);
                        w[j] = ptx::pack_bf16x2(ga * acc[32 + 2 * j], gb * acc[33 + 2 * j]);
                    }
                    staging_free();
                    stage_row_bf16(stage, lane, w);
                    send(col / 4, row0, rows_inside && col < p.N);
                } else {
                    if constexpr (FORM == BF16_PLAIN) {
#pragma unroll
                        for (int h = 0; h < C::kPiece; h += 32) {
                            if (col + h >= p.tail_col) {
                                if (mine) {
                                    float *dst = p.tail + static_cast<long long>(row0 + lane) * p.tail_pitch + (col + h - p.tail_col);
#pragma unroll
                                    for (int j = 0; j < 32; ++j)
                                        if (col + h + j < p.N) dst[j] = acc[h + j];
                                }
                            } else if (col + h < p.silu_cols) {
#pragma unroll
                                for (int j = 0; j < 32; ++j) acc[h + j] = silu_fast(acc[h + j]);
                            }
                        }
                    } else {
                        const uint4 *f = reinterpret_cast<const uint4 *>(p.factor + (mine ? static_cast<long long>(p.factor_rows[row0 + lane]) * p.factor_pitch : 0) + col);
#pragma unroll
                        for (int o = 0; o < C::kPiece / 8; ++o) {
                            const uint4 x4 = mine && col + 8 * o < p.N ? __ldg(f + o) : make_uint4(0u, 0u, 0u, 0u);   // N is a multiple of 8
                            const uint32_t x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                acc[8 * o + 2 * i] = gelu_tanh(acc[8 * o + 2 * i]) * bf16_lo(x[i]);
                                acc[8 * o + 2 * i + 1] = gelu_tanh(acc[8 * o + 2 * i + 1]) * bf16_hi(x[i]);
                            }
                        }
                    }
                    if (FORM != BF16_PLAIN || col < p.tail_col) {
                        staging_free();
                        uint32_t w[C::kPiece / 2];
#pragma unroll
                        for (int j = 0; j < C::kPiece / 2; ++j) w[j] = ptx::pack_bf16x2(acc[2 * j], acc[2 * j + 1]);
                        if constexpr (C::kPiece == 64) {
#pragma unroll
                            for (int j = 0; j < 8; ++j) ptx::sts128(stage + lane * 128 + ((j ^ (lane & 7)) << 4), w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
                        } else {
                            stage_row_bf16(stage, lane, w);
                        }
                        send(col / 2, row0, rows_inside && col < p.N);
                    }
                }
#pragma unroll
                for (int j = 0; j + C::kPiece < C::kCols; ++j) acc[j] = acc[j + C::kPiece];
            }
        }
        if (lane == 0) ptx::tma_store_wait_all<0>();
        __syncwarp();
    }

    // ---------------------------------------------------------------- teardown
    ptx::tc_fence_before();
    __syncthreads();
    if (*abort_flag) {   // a wait ran out: copies still in flight get time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::cluster_sync();   // neither CTA leaves while the other can still signal its barriers
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

}  // namespace gptb200
