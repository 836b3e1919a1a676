// Products of 9 to 64 rows of fp32 with a weight matrix stored [k][n] (linear layers) or [n][k] (un-embedding, grad_x): y[m][n] = x[m][k] . w, bias and GELU,
// on the tensor cores and no less exact than fp32 FMAs.
//
// Both operands are split exactly into three bf16 values a0 + a1 + a2 (8 + 8 + 8 bits: the first truncated, the others rounded, so |a1| < 2^-7 |a| and |a2| <=
// 2^-15 |a|), and all of their products but a2 . b2 (2^-30) are added.  The tensor core adds into its accumulator with truncation, so the accumulator is handed to
// fp32 sums in registers (round to nearest) after every step of 16 k, the exact products a0 . b0 apart from the others.  Off from 64-bit sums, this / fp32 FMAs, of
// the result's size: k 32, n 8192 4.5e-8 / 6.9e-8, 768 x 2304 8.3e-8 / 1.15e-7, 3072 x 768 1.08e-7 / 1.54e-7, 768 x 50304 1.33e-7 / 2.08e-7; sums of a single
// product at most 6.0e-8 / 5.9e-8, where six products in one accumulator were off by 2.3e-7 (us: output layer at 64 rows 59.5, then 50; at 9 rows 35.0 and 33.0).
// An infinite value splits into parts that are NaN: outputs that come out as NaN are computed again with fp32 FMAs at the end, so that they are infinite or NaN
// as there.
//
// A block computes 128 columns for all rows over its share of k.  The weights are the M = 128 operand; split, they never go back to shared memory: the converter
// warps write them to TMEM, where the instructions take their A operand from.
//   warps 0-7    converters: 16 k of the landed tile (lane = column) -> three bf16 pairs of 8 TMEM columns; the two groups of four alternate
//   warps 8-15   sums: accumulator -> registers, half of the rows each
//   warps 16-19  x: global -> three bf16 tiles of 64 k in shared memory (B operand)
//   warp 20      TMA producer: 32 KB of weights per 64 k, four stages
//   warps 21, 22 issue the instructions, every other step each: one of them took 500 cycles per step for its waits, instructions (six then) and commits (output layer
//                55 us at 64 rows and 40 at 9; two 47 and 33, three 47 and 32).  More converters, or the instructions of several steps in turn, were slower.
// The un-embedding has enough column tiles for all SMs (blocks walk over them); narrow layers share k in a cluster, partial tiles meet in rank order through
// distributed shared memory.
#pragma once

#include <cooperative_groups.h>

#include "gemm_sm100.cuh"

namespace gptb200 {

constexpr int kRowsIssuers = 2;
constexpr int kRowsThreads = (21 + kRowsIssuers) * 32;
constexpr int kRowsStages = 4, kRowsStageBytes = 128 * 64 * 4;
constexpr int kRowsSlotCols = 24;                      // split weights of 16 k: 3 x 8 TMEM columns
constexpr int kRowsMaxSlots = 8, kRowsMaxAccs = 4;
constexpr int kRowsXBufs = 2;

struct RowsParams {
    float *y, *act;            // act: null, or gelu(y)
    const float *x, *w, *bias; // bias: null for none
    int M, N, K;
    int slice;                 // k per block of a cluster, a multiple of 16
    int tiles;                 // of 128 columns
    int *status;
    int early;                 // weights may be read before the predecessor on the stream has completed
};

// TMEM of a block: accumulators (with two of them the way to the sums and back was what a step took), then split weights.
template <int MR>
struct RowsTmem {
    static constexpr int kAccs = MR == 64 ? 3 : 4, kSlots = MR == 64 ? 5 : 8;
    static constexpr int kRest = MR < 32 ? 32 : MR, kAccCols = 2 * kRest;   // leading products, and the others kRest columns on
    static constexpr int kSlotBase = kAccs * kAccCols;
    static_assert(kAccs <= kRowsMaxAccs && kSlots <= kRowsMaxSlots && kSlotBase + kSlots * kRowsSlotCols <= 512, "TMEM");
};

constexpr int rows_smem_bytes(int mr) { return kRowsStages * kRowsStageBytes + kRowsXBufs * 3 * mr * 128 + 1024 + 512; }

namespace rows {

// Two neighbours in k -> their three bf16 pairs (the first value in the low half).
__device__ __forceinline__ void split3(float a, float b, uint32_t &p0, uint32_t &p1, uint32_t &p2)
{
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    p0 = __byte_perm(ua, ub, 0x7632);
    const float ra = a - __uint_as_float(ua & 0xFFFF0000u), rb = b - __uint_as_float(ub & 0xFFFF0000u);
    p1 = ptx::pack_bf16x2(ra, rb);
    p2 = ptx::pack_bf16x2(ra - bf16_lo(p1), rb - bf16_hi(p1));
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]),
                 "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t *v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr) : "memory");
}

// A from TMEM (lane = row of A, a column = two neighbours in k), B from shared memory.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "setp.ne.b32 P, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, P;\n\t}"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// One step's eight products, the smallest first: split weights at TMEM columns `a`, the parts of x `part` bytes apart.  The leading products go to `d`, the others to
// `rest`, or all of them to one accumulator.
__device__ __forceinline__ void issue_step(uint32_t d, uint32_t rest, uint32_t a, const ptx::SmemDesc &x, uint32_t at, uint32_t part, uint32_t idesc)
{
    mma_ts(rest, a + 16, x.at(at + part), idesc, 0u);
    mma_ts(rest, a + 8, x.at(at + 2 * part), idesc, 1u);
    mma_ts(rest, a + 16, x.at(at), idesc, 1u);
    mma_ts(rest, a, x.at(at + 2 * part), idesc, 1u);
    mma_ts(rest, a + 8, x.at(at + part), idesc, 1u);
    mma_ts(rest, a + 8, x.at(at), idesc, 1u);
    mma_ts(rest, a, x.at(at + part), idesc, 1u);
    mma_ts(d, a, x.at(at), idesc, d == rest ? 1u : 0u);
}

}  // namespace rows

// Walk over the steps of 16 k of a block's tiles; every role takes it alike.
struct RowsWalk {
    int steps, blocks;      // of 16 k, of 64 k
    int k0;
    __device__ __forceinline__ RowsWalk(const RowsParams &p, int rank)
    {
        k0 = rank * p.slice;
        steps = max(0, (min(p.K, k0 + p.slice) - k0 + 15) / 16);
        blocks = (steps + 3) / 4;
    }
    __device__ __forceinline__ int in_block(int b) const { return min(4, steps - 4 * b); }
};

// grid (column tiles, or blocks that walk over them; cluster over k)
template <int MR, bool W_NK>
__global__ void __launch_bounds__(kRowsThreads, 1)
rows_tensor_kernel(const __grid_constant__ CUtensorMap tmap_w, const RowsParams p)
{
    namespace cg = cooperative_groups;
    using T = RowsTmem<MR>;
    constexpr int kXBytes = 3 * MR * 128, kCols = MR / 2;
    constexpr uint32_t kIdesc = ptx::make_idesc_bf16(128, MR, false, false);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    const uint32_t x_base = smem_base + kRowsStages * kRowsStageBytes;
    const uint32_t bar_base = x_base + kRowsXBufs * kXBytes;
    auto w_full = [&](int s) { return bar_base + 8u * s; };
    auto w_empty = [&](int s) { return bar_base + 8u * (kRowsStages + s); };
    auto a_full = [&](int r) { return bar_base + 8u * (2 * kRowsStages + r); };
    auto done = [&](int r) { return bar_base + 8u * (2 * kRowsStages + kRowsMaxSlots + r); };      // a step's instructions: its sums are there, its weights read
    constexpr int kX = 2 * kRowsStages + 2 * kRowsMaxSlots;
    auto x_full = [&](int b) { return bar_base + 8u * (kX + b); };
    auto x_empty = [&](int b) { return bar_base + 8u * (kX + kRowsXBufs + b); };
    auto acc_empty = [&](int b) { return bar_base + 8u * (kX + 2 * kRowsXBufs + b); };
    const uint32_t drain_bar = bar_base + 8u * (kX + 2 * kRowsXBufs + kRowsMaxAccs);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + (bar_base - smem_base) + 8 * (kX + 2 * kRowsXBufs + kRowsMaxAccs + 1));
    static_assert(8 * (kX + 2 * kRowsXBufs + kRowsMaxAccs + 1) + 12 <= 512, "barriers");
    volatile uint32_t *abort_flag = tmem_slot + 1, *nan_flag = tmem_slot + 2;

    const int warp = ptx::warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int S = gridDim.y, rank = blockIdx.y;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRowsStages; ++s) {
            ptx::mbar_init(w_full(s), 1);
            ptx::mbar_init(w_empty(s), 8);
        }
        for (int r = 0; r < T::kSlots; ++r) {
            ptx::mbar_init(a_full(r), 4);
            ptx::mbar_init(done(r), 1);
        }
        for (int b = 0; b < kRowsXBufs; ++b) {
            ptx::mbar_init(x_full(b), 4);
            ptx::mbar_init(x_empty(b), kRowsIssuers);
        }
        for (int b = 0; b < T::kAccs; ++b) ptx::mbar_init(acc_empty(b), 8);
        ptx::mbar_init(drain_bar, kRowsIssuers);
        *abort_flag = *nan_flag = 0u;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_w);
    }
    if (warp == 21) {
        ptx::tmem_alloc(ptx::smem_u32(tmem_slot), 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = ptx::warp_uniform(*tmem_slot);
    const RowsWalk walk(p, rank);
    if (!p.early) grid_dependency_wait();
    bool ok = true;

    if (warp < 8) {
        // ------------------------------------------------------------ converters
        const int set = warp >> 2, quarter = warp & 3, n = quarter * 32 + lane;
        const uint32_t slots = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + T::kSlotBase;
        uint32_t g = 0, s = 0, ph = 0;
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            for (int b = 0; ok && b < walk.blocks; ++b) {
                if (!bounded_wait(w_full(s), ph, abort_flag, p.status, DEV_TIMEOUT_CONVERT)) {
                    ok = false;
                    break;
                }
                const uint32_t stage = smem_base + s * kRowsStageBytes;
                const int steps = walk.in_block(b);
                for (int ks = 0; ks < steps; ++ks, ++g) {
                    if (static_cast<int>(g & 1u) != set) continue;
                    float v[16];
                    if (W_NK) {   // boxes of 32 k: [128 columns][32 k], 16-byte pieces XOR-ed with the column mod 8
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 f = ptx::lds128(stage + (ks >> 1) * 16384 + n * 128 + ((((ks & 1) * 4 + j) ^ (n & 7)) << 4));
                            v[4 * j] = f.x;
                            v[4 * j + 1] = f.y;
                            v[4 * j + 2] = f.z;
                            v[4 * j + 3] = f.w;
                        }
                    } else {      // [64 k][128 columns]
                        const float *w = reinterpret_cast<const float *>(smem_gen + s * kRowsStageBytes) + ks * 16 * 128 + n;
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = w[j * 128];
                    }
                    uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) rows::split3(v[2 * j], v[2 * j + 1], p0[j], p1[j], p2[j]);
                    const uint32_t r = g % T::kSlots;
                    if (!bounded_wait(done(r), ((g / T::kSlots) & 1u) ^ 1u, abort_flag, p.status, DEV_TIMEOUT_CONVERT)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    rows::tmem_st8(slots + r * kRowsSlotCols, p0);
                    rows::tmem_st8(slots + r * kRowsSlotCols + 8, p1);
                    rows::tmem_st8(slots + r * kRowsSlotCols + 16, p2);
                    rows::tmem_st_wait();
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(a_full(r));
                }
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(w_empty(s));
                if (++s == kRowsStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp < 16) {
        // ------------------------------------------------------------ sums
        const int half = (warp - 8) >> 2, quarter = warp & 3, n = quarter * 32 + lane;
        const uint32_t mine = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + half * kCols;
        uint32_t g = 0;
        if (p.early) grid_dependency_wait();   // y may still be read by it
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            float acc[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j) acc[j] = 0.0f;
            for (int ks = 0; ks < walk.steps; ++ks, ++g) {
                const uint32_t b = g % T::kAccs;
                if (!bounded_wait(done(g % T::kSlots), (g / T::kSlots) & 1u, abort_flag, p.status, DEV_TIMEOUT_EPILOGUE)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                constexpr int kPiece = kCols < 16 ? kCols : 16;
#pragma unroll
                for (int c = 0; c < kCols; c += kPiece) {
                    uint32_t v[kPiece], u[kPiece];
#pragma unroll
                    for (int j = 0; j < kPiece; j += 8) {
                        rows::tmem_ld8(mine + b * T::kAccCols + c + j, v + j);
                        rows::tmem_ld8(mine + b * T::kAccCols + T::kRest + c + j, u + j);
                    }
                    ptx::tmem_ld_wait();
                    if (c + kPiece == kCols) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(acc_empty(b));
                    }
#pragma unroll
                    for (int j = 0; j < kPiece; ++j) acc[c + j] += __uint_as_float(v[j]) + __uint_as_float(u[j]);
                }
            }
            if (!ok) break;
            if (S == 1) {
                const int col = t * 128 + n;
                if (col < p.N) {
                    const float bias = p.bias ? __ldg(p.bias + col) : 0.0f;
                    float all = 0.0f;
#pragma unroll
                    for (int j = 0; j < kCols; ++j) {
                        const int m = half * kCols + j;
                        all += acc[j];
                        if (m < p.M) {
                            const float v = acc[j] + bias;
                            p.y[static_cast<long long>(m) * p.N + col] = v;
                            if (p.act) p.act[static_cast<long long>(m) * p.N + col] = gelu_tanh(v);
                        }
                    }
                    if (isnan(all)) *nan_flag = 1u;
                }
            } else {   // the partial tile [row][column] takes the place of the weights: all of them have been converted
                float *tile = reinterpret_cast<float *>(smem_gen);
#pragma unroll
                for (int j = 0; j < kCols; ++j) tile[(half * kCols + j) * 128 + n] = acc[j];
            }
        }
    } else if (warp < 20) {
        // ------------------------------------------------------------ x
        if (p.early) grid_dependency_wait();
        if (threadIdx.x == 16 * 32) grid_dependency_launch();
        constexpr int kUnits = MR * 8 / 128;   // of 8 k per thread
        const int tid = threadIdx.x - 16 * 32;
        uint32_t xb = 0, ph = 0;
        float4 v[kUnits][2];
        auto fetch = [&](int b) {
#pragma unroll
            for (int u = 0; u < kUnits; ++u) {
                const int i = tid + u * 128, row = i >> 3, k = walk.k0 + b * 64 + (i & 7) * 8;
                const float4 *src = reinterpret_cast<const float4 *>(p.x + static_cast<long long>(row) * p.K + k);
                v[u][0] = row < p.M && k < p.K ? __ldg(src) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);          // K is a multiple of 4
                v[u][1] = row < p.M && k + 4 < p.K ? __ldg(src + 1) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        };
        if (walk.blocks > 0) fetch(0);
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            for (int b = 0; b < walk.blocks; ++b) {
                if (!bounded_wait(x_empty(xb), ph ^ 1u, abort_flag, p.status, DEV_TIMEOUT_CONVERT)) {
                    ok = false;
                    break;
                }
                const uint32_t dst = x_base + xb * kXBytes;
#pragma unroll
                for (int u = 0; u < kUnits; ++u) {
                    const int i = tid + u * 128, row = i >> 3, c = i & 7;
                    const float f[8] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w, v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
                    uint32_t p0[4], p1[4], p2[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) rows::split3(f[2 * j], f[2 * j + 1], p0[j], p1[j], p2[j]);
                    const uint32_t at = dst + row * 128 + ((c ^ (row & 7)) << 4);
                    ptx::sts128(at, p0[0], p0[1], p0[2], p0[3]);
                    ptx::sts128(at + MR * 128, p1[0], p1[1], p1[2], p1[3]);
                    ptx::sts128(at + 2 * MR * 128, p2[0], p2[1], p2[2], p2[3]);
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(x_full(xb));
                fetch(b + 1 < walk.blocks ? b + 1 : 0);   // the next block, or the next tile's first
                if (++xb == kRowsXBufs) {
                    xb = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 20) {
        // ------------------------------------------------------------ TMA producer
        const bool issuer = ptx::elect_one();
        uint32_t s = 0, ph = 0;
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            for (int b = 0; b < walk.blocks; ++b) {
                if (!bounded_wait(w_empty(s), ph ^ 1u, abort_flag, p.status, DEV_TIMEOUT_PRODUCER)) {
                    ok = false;
                    break;
                }
                if (issuer) {
                    const int boxes = (walk.in_block(b) + 1) / 2, k = walk.k0 + b * 64;   // of 32 k
                    ptx::mbar_arrive_expect_tx(w_full(s), boxes * 16384);
                    for (int i = 0; i < boxes; ++i) {
                        const uint32_t dst = smem_base + s * kRowsStageBytes + i * 16384;
                        if (W_NK)
                            ptx::tma_load_2d(dst, &tmap_w, k + 32 * i, t * 128, w_full(s));
                        else
                            ptx::tma_load_2d(dst, &tmap_w, t * 128, k + 32 * i, w_full(s));
                    }
                }
                __syncwarp();
                if (++s == kRowsStages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else {
        // ------------------------------------------------------------ instructions
        const bool issuer = ptx::elect_one();
        const ptx::SmemDesc desc_x = ptx::smem_desc_words(x_base, 16, 1024, ptx::kLayoutSw128);
        uint32_t g = 0, xb = 0, ph = 0;
        const uint32_t turn = warp - 21;
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            for (int b = 0; ok && b < walk.blocks; ++b) {
                if (!bounded_wait(x_full(xb), ph, abort_flag, p.status, DEV_TIMEOUT_MMA_FULL)) {
                    ok = false;
                    break;
                }
                const int steps = walk.in_block(b);
                for (int ks = 0; ks < steps; ++ks, ++g) {
                    if (g % kRowsIssuers != turn) continue;
                    const uint32_t buf = g % T::kAccs, r = g % T::kSlots;
                    if (!bounded_wait(acc_empty(buf), ((g / T::kAccs) & 1u) ^ 1u, abort_flag, p.status, DEV_TIMEOUT_MMA_TMEM) ||
                        !bounded_wait(a_full(r), (g / T::kSlots) & 1u, abort_flag, p.status, DEV_TIMEOUT_MMA_CONV)) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t d = tmem + buf * T::kAccCols, a = tmem + T::kSlotBase + r * kRowsSlotCols, x = xb * kXBytes + ks * 32;
                    if (issuer) {
                        rows::issue_step(d, d + T::kRest, a, desc_x, x, MR * 128, kIdesc);
                        ptx::mma_commit(done(r));
                    }
                }
                if (issuer) ptx::mma_commit(x_empty(xb));
                if (++xb == kRowsXBufs) {
                    xb = 0;
                    ph ^= 1u;
                }
            }
        }
        if (issuer) ptx::mma_commit(drain_bar);   // TMEM is about to be released
        bounded_wait(drain_bar, 0u, abort_flag, p.status, DEV_TIMEOUT_DRAIN);
        __syncwarp();
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (*abort_flag) {   // a wait ran out: copies still in flight get time to land
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    if (warp == 21) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
    bool nan_seen = *nan_flag != 0u;
    if (S > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        // rank order; this block finishes every S-th run of four-column pieces
        float *tile = reinterpret_cast<float *>(smem_gen);
        for (int e = rank * kRowsThreads + threadIdx.x; e < p.M * 32; e += S * kRowsThreads) {
            const int m = e >> 5, col = blockIdx.x * 128 + 4 * (e & 31);
            if (col >= p.N) continue;
            float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int q0 = 0; q0 < S; q0 += 8) {   // up to eight remote loads in flight
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    v[j] = q0 + j < S ? reinterpret_cast<const float4 *>(cluster.map_shared_rank(tile, q0 + j))[e] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    sum.x += v[j].x;
                    sum.y += v[j].y;
                    sum.z += v[j].z;
                    sum.w += v[j].w;
                }
            }
            if (p.bias) {   // need not be 16-byte aligned
                sum.x += __ldg(p.bias + col);
                sum.y += __ldg(p.bias + col + 1);
                sum.z += __ldg(p.bias + col + 2);
                sum.w += __ldg(p.bias + col + 3);
            }
            *reinterpret_cast<float4 *>(p.y + static_cast<long long>(m) * p.N + col) = sum;
            if (p.act) *reinterpret_cast<float4 *>(p.act + static_cast<long long>(m) * p.N + col) = make_float4(gelu_tanh(sum.x), gelu_tanh(sum.y), gelu_tanh(sum.z), gelu_tanh(sum.w));
            nan_seen |= isnan(sum.x + sum.y + sum.z + sum.w);
        }
        cluster.sync();   // no block leaves while its tile may still be read
    }
    if (nan_seen) {
        // rare and slow, but no work for the loops above: the four columns of a piece one after the other
        for (int t = blockIdx.x; t < p.tiles; t += gridDim.x)
            for (int e = rank * kRowsThreads + threadIdx.x; e < p.M * 32; e += S * kRowsThreads)
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {
                    const int m = e >> 5, col = t * 128 + 4 * (e & 31) + c;
                    const long long at = static_cast<long long>(m) * p.N + col;
                    if (col >= p.N || !isnan(p.y[at])) continue;
                    const float *x = p.x + static_cast<long long>(m) * p.K, *w = W_NK ? p.w + static_cast<long long>(col) * p.K : p.w + col;
                    const long long step = W_NK ? 1 : p.N;
                    float sum = 0.0f;
#pragma unroll 1
                    for (int k = 0; k < p.K && !isnan(sum); k += 4) {   // K is a multiple of 4
                        const float4 v = __ldcg(reinterpret_cast<const float4 *>(x + k));
                        const float u[4] = {w[k * step], w[(k + 1) * step], w[(k + 2) * step], w[(k + 3) * step]};
                        sum = fmaf(v.w, u[3], fmaf(v.z, u[2], fmaf(v.y, u[1], fmaf(v.x, u[0], sum))));
                    }
                    if (p.bias) sum += __ldg(p.bias + col);
                    p.y[at] = sum;
                    if (p.act) p.act[at] = gelu_tanh(sum);
                }
    }
}

}  // namespace gptb200
