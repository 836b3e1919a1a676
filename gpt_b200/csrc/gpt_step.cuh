// Kernels of a GPT-2 generation step in one launch.
//
// As one launch per operator a step of 12 layers is a chain of 89 launches of 3 - 16 us for 0.5 GB of weights (75 us of HBM
// time): bound by launches, not by memory.  Here one block per SM stays for the whole step.  Phases meet at grid barriers
// (arrivals counted in device memory, a cooperative launch keeps all blocks resident), and while a block waits at one its weights of the
// next phase are already on their way: they depend on nothing.  Arithmetic is fp32 FMAs, the products of 16 padded rows and more three bf16 parts per operand
// on the tensor cores with fp32 sums; sums have a fixed order.
#pragma once

#include <cfloat>
#include <cuda_runtime.h>

#include "gemm_sm100.cuh"  // gelu_tanh
#include "rows_sm100.cuh"  // products in three bf16 parts
#include "gpt_step.h"

namespace gptb200 {
namespace step {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kCols = 64;                    // output columns per item
constexpr int kBody = 8;                     // 16-byte weight loads in flight per thread: 256 k-rows of an item
constexpr unsigned kPollLimit = 1u << 22;    // some seconds; reached only if a block of the grid never ran

// Grid barrier in two halves, so that loads can be issued between them.  The counter only grows: `target` is what it reads once all
// blocks have arrived at this barrier.
__device__ __forceinline__ void arrive(const GptStep &s, unsigned &target)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(s.sync) : "memory");
    }
    target += gridDim.x;
}

// A wait that runs out sets `gave_up` (thread 0's).  The block waits at no later barrier then, and goes on to the end of the step with whatever sums it
// finds: it writes neither logits nor position, and the keys and values that it writes lie behind the last valid position.  (Leaving at once, by a
// __syncthreads_or in every barrier, made a step of one sequence 4 us longer and one of 32 14 us.)
__device__ __forceinline__ void await(const GptStep &s, unsigned target, bool &gave_up, unsigned limit = kPollLimit)
{
    if (threadIdx.x == 0 && !gave_up) {
        unsigned seen = 0, tries = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(s.sync) : "memory");
            if (tries++ == limit) {
                gave_up = true;
                atomicExch(s.sync + 2, 1u);
                atomicCAS(s.status, 0, DEV_TIMEOUT_GRID);
                break;
            }
        } while (static_cast<int>(seen - target) < 0);
    }
    __syncthreads();
}

// Whether a barrier of this generation ran out in an earlier launch: the counter is short of arrivals then, and no launch can wait on it until the
// cache is filled anew.  For thread 0 of a block.
__device__ __forceinline__ bool lost(const GptStep &s)
{
    const bool is = *reinterpret_cast<volatile unsigned *>(s.sync + 2) != 0;
    if (is) atomicCAS(s.status, 0, DEV_TIMEOUT_GRID);
    return is;
}

// Self-test: a barrier that all blocks of a grid of one reach, one that nothing reaches, and what that leaves behind.
static __global__ void barrier_selftest_kernel(const GptStep s, unsigned limit)
{
    unsigned target = 0;
    bool gave_up = false;
    arrive(s, target);
    await(s, target, gave_up, limit);
    const bool early = gave_up;
    await(s, target + 1, gave_up, limit);
    if (threadIdx.x == 0 && (early || !gave_up || !lost(s))) atomicExch(s.status, DEV_TIMEOUT_SELFTEST);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s)))); }

// Sum of N values, neighbours first: log2 N roundings deep.  One value after the other made the logits' error against 64 bits larger than that of the
// step that runs operator by operator (GPT-2 124M, one sequence: 3.47e-7 of their size against 3.34e-7; 3.27e-7 so, in the same time).
template <int N>
__device__ __forceinline__ float4 pairwise(float4 (&v)[N])
{
#pragma unroll
    for (int w = 1; w < N; w *= 2)
#pragma unroll
        for (int i = 0; i + w < N; i += 2 * w) v[i] = add4(v[i], v[i + w]);
    return v[0];
}
template <int N>
__device__ __forceinline__ float pairwise(float (&v)[N])
{
#pragma unroll
    for (int w = 1; w < N; w *= 2)
#pragma unroll
        for (int i = 0; i + w < N; i += 2 * w) v[i] += v[i + w];
    return v[0];
}

// Sum of the slices' partial sums at one position, in a fixed order; `stride` floats between slices.  Written by other blocks of this launch: read from L2.
template <int FLIGHT = 12>
__device__ __forceinline__ float4 sum_parts4(const float *p, int splits, int stride)
{
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (; splits > 0; splits -= FLIGHT) {   // loads in flight: one L2 round trip for what the plan makes of GPT-2
        float4 v[FLIGHT];
#pragma unroll
        for (int i = 0; i < FLIGHT; ++i, p += stride)
            v[i] = i < splits ? __ldcg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        sum = add4(sum, pairwise(v));
    }
    return sum;
}

__device__ __forceinline__ float sum_parts(const float *p, int splits, int stride)
{
    float sum = 0.0f;
#pragma unroll 1
    for (; splits > 0; splits -= 4) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i, p += stride) v[i] = i < splits ? __ldcg(p) : 0.0f;
        sum += pairwise(v);
    }
    return sum;
}

// ---- one or two rows --------------------------------------------------------------------------------------------------------
// Weights go straight to registers: thread (krow, lane16) of an item reads 16 bytes of k-rows krow, krow + 32, ... (a half-warp 256
// contiguous bytes), all of a slice of up to 256 rows at once, before the barrier in front of the phase.  GPT-2 124M on 148 SMs: 144 items
// in every phase.  Every block keeps the whole residual stream in shared memory and norms it itself (bitwise the same everywhere), and the
// blocks of one head compute its attention once each: four barriers per layer instead of seven.  A phase lasts one to two
// microseconds, so what 16 warps issue counts as much as what they wait for: addresses are worked out once per launch (Share), and
// warps without data skip (with both left out a step of GPT-2 124M took 270 us).  One row at position 64 - 96: 223 us per step, against 435 us as
// 89 launches (a prompt of 64 tokens and 32 steps: 8.6 ms, was 15.7 - 16.2).  What is left is the length of the chain: at a barrier 1.1 us
// between the last arrival and the first use of its data, then up to 1.5 us for 148 blocks that read the same 36 KB of partial sums.
// Tried: the next phase's weights towards L2 while a phase computes (0.15 ms slower: their traffic delays the partial sums); clusters of two blocks that
// each read half of the partial sums (no faster).

// A thread's part of an item.
struct Share {
    int offset;     // of its first weight
    int count;      // its k-rows, 32 apart
    int k0, rows;   // the item's slice
    int split, col;   // col: of the item
};

__device__ __forceinline__ Share share_of(const StepPhase &ph, int item)
{
    Share r;
    r.split = item / ph.groups;
    r.col = (item - r.split * ph.groups) * kCols;
    r.k0 = r.split * ph.slice;
    r.rows = item < ph.groups * ph.splits ? min(ph.K - r.k0, ph.slice) : 0;
    const int krow = threadIdx.x >> 4, col = r.col + (threadIdx.x & 15) * 4;
    r.offset = (r.k0 + krow) * ph.N + col;
    r.count = col < ph.N ? max(0, (r.rows - krow + 31) >> 5) : 0;
    return r;
}

__device__ __forceinline__ void fetch(float4 (&wv)[kBody], const float *w, const StepPhase &ph, const Share &r, int done = 0)
{
    const float *p = w + r.offset + static_cast<size_t>(done * 32) * ph.N;
    const int stride = 32 * ph.N;
#pragma unroll
    for (int j = 0; j < kBody; ++j, p += stride)
        wv[j] = done + j < r.count ? __ldcs(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// part[split][m][col ..] = xs[m][.] . w over the item's slice.  wv holds the first weights; red: [kWarps][MR][kCols].
template <int MR>
__device__ __forceinline__ void item_product(float4 (&wv)[kBody], const float *w, const StepPhase &ph, const Share &r, const float *xs, int pitch, float *red, float *part)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float *x = xs + (threadIdx.x >> 4);
    float acc[MR][4] = {};
#pragma unroll 1
    for (int done = 0; done * 32 < r.rows; done += kBody, x += 32 * kBody) {
        if (done > 0) fetch(wv, w, ph, r, done);
#pragma unroll
        for (int j = 0; j < kBody; ++j)
            if (done + j < r.count) {
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    const float v = x[m * pitch + 32 * j];
                    acc[m][0] = fmaf(v, wv[j].x, acc[m][0]);
                    acc[m][1] = fmaf(v, wv[j].y, acc[m][1]);
                    acc[m][2] = fmaf(v, wv[j].z, acc[m][2]);
                    acc[m][3] = fmaf(v, wv[j].w, acc[m][3]);
                }
            }
    }
#pragma unroll
    for (int m = 0; m < MR; ++m) {
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][c] += __shfl_xor_sync(0xffffffffu, acc[m][c], 16);
        if (lane < 16) *reinterpret_cast<float4 *>(red + (warp * MR + m) * kCols + lane * 4) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
    }
    __syncthreads();
    if (threadIdx.x < MR * kCols) {
        const int m = threadIdx.x / kCols, col = r.col + threadIdx.x % kCols;
        float v[kWarps];
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v[i] = red[i * MR * kCols + threadIdx.x];
        if (col < ph.N) part[(r.split * MR + m) * ph.N + col] = pairwise(v);
    }
}

// Count, mean and sum of squared distances from it of the values that a warp's threads hold, for each warp with any.
// The threads of one row are kThreads / MR consecutive ones.
template <int MR>
__device__ __forceinline__ void warp_moments(const float *row, int d, float4 *part)
{
    constexpr int kPer = kThreads / MR;
    const int at = (threadIdx.x % kPer) * 4, lane = threadIdx.x & 31;
    if (at - lane * 4 >= d) return;
    float sum = 0.0f, n = 0.0f, var = 0.0f;
#pragma unroll 1
    for (int i = at; i < d; i += kPer * 4) {
        const float4 v = *reinterpret_cast<const float4 *>(row + i);
        sum += (v.x + v.y) + (v.z + v.w);
    }
#pragma unroll 1
    for (int i = at - lane * 4; i < d; i += kPer * 4) n += static_cast<float>(min(d - i, 128));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / n;
#pragma unroll 1
    for (int i = at; i < d; i += kPer * 4) {
        const float4 v = *reinterpret_cast<const float4 *>(row + i);
        const float a = v.x - mean, b = v.y - mean, c = v.z - mean, e = v.w - mean;
        var += (a * a + b * b) + (c * c + e * e);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) var += __shfl_xor_sync(0xffffffffu, var, o);
    if (lane == 0) part[threadIdx.x >> 5] = make_float4(n, mean, var, 0.0f);
}

// Mean and standard deviation of every row from the warps' moments: mean of the means, distances of the means added to the squares.
template <int MR>
__device__ __forceinline__ void row_statistics(const float4 *part, int d, float (&mean)[MR], float (&sd)[MR])
{
    constexpr int kPer = kWarps / MR;
    const int warps = min((d + 127) >> 7, kPer);
#pragma unroll
    for (int m = 0; m < MR; ++m) {
        float sum = 0.0f, var = 0.0f;
        for (int w = 0; w < warps; ++w) sum = fmaf(part[m * kPer + w].x, part[m * kPer + w].y, sum);
        mean[m] = sum / d;
        for (int w = 0; w < warps; ++w) {
            const float4 v = part[m * kPer + w];
            var += fmaf(v.x * (v.y - mean[m]), v.y - mean[m], v.z);
        }
        sd[m] = sqrtf(var / d + 1e-5f);
    }
}

// The largest shared memory of the kernel below, in floats.
inline size_t small_shared_floats(int mr, int d, int hd, int max_len, int widest)
{
    return size_t(mr) * d + size_t(mr) * widest + size_t(kWarps) * mr * kCols + size_t(mr) * 3 * hd + size_t(kWarps) * (hd + 4) + size_t(mr) * max_len;
}

// MR: the sequences.
template <int MR>
__global__ void __launch_bounds__(kThreads, 1)
gpt_step_kernel(const GptStep s, int widest)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ float4 moments[kWarps];
    float *res = sm;                                 // [MR][d] residual stream
    float *xs = res + MR * s.d;                      // [MR][widest] activations of an item
    float *red = xs + MR * widest;                   // [kWarps][MR][kCols]
    float *fresh = red + kWarps * MR * kCols;        // [MR][3][hd] new q, k, v of a head
    float *out = fresh + MR * 3 * s.hd;              // [kWarps][hd + 4] parts of a head's output, and of its weights' sum
    float *prob = out + kWarps * (s.hd + 4);         // [MR][max_len]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = s.d;
    const int p = *s.pos;
    if (p < 0 || p >= s.max_len || p >= s.max_pos) return;   // all blocks alike
    bool gave_up = tid == 0 && lost(s);
    unsigned target = s.sync[1];
    const int first = blockIdx.x;                    // this block's first item of every phase
    const Share of_qkv = share_of(s.qkv, first), of_proj = share_of(s.proj, first), of_up = share_of(s.up, first), of_down = share_of(s.down, first);
    float4 wv[kBody];
    fetch(wv, s.qkv_w, s.qkv, of_qkv);

    constexpr int kPer = kThreads / MR;   // threads of a row
    const int mine = tid / kPer, at4 = (tid % kPer) * 4;
#pragma unroll 1
    for (int c = at4; c < d; c += kPer * 4)
        *reinterpret_cast<float4 *>(res + mine * d + c) = add4(__ldg(reinterpret_cast<const float4 *>(s.wte + static_cast<size_t>(s.tokens[mine]) * d + c)),
                                                               __ldg(reinterpret_cast<const float4 *>(s.wpe + static_cast<size_t>(p) * d + c)));
    warp_moments<MR>(res + mine * d, d, moments);
    if (__syncthreads_or(gave_up)) return;

    // res += the finished product, with the moments of the new rows
    auto add_result = [&](const float *part, const StepPhase &ph, const float *bias) {
#pragma unroll 1
        for (int c = at4; c < d; c += kPer * 4) {
            const float4 be = __ldg(reinterpret_cast<const float4 *>(bias + c));
            const float4 v = add4(sum_parts4(part + mine * d + c, ph.splits, MR * d), be);
            *reinterpret_cast<float4 *>(res + mine * d + c) = add4(*reinterpret_cast<const float4 *>(res + mine * d + c), v);
        }
        warp_moments<MR>(res + mine * d, d, moments);
        __syncthreads();
    };
    // a product behind a norm of the residual stream
    // (gain0, bias0: the norm's parameters of the first item's k-row `tid`, loaded like its weights before the barrier)
    float gain0 = 0.0f, bias0 = 0.0f;
    auto fetch_norm = [&](const Share &r, const float *gain, const float *bias) {
        if (tid < r.rows) {
            gain0 = __ldg(gain + r.k0 + tid);
            bias0 = __ldg(bias + r.k0 + tid);
        }
    };
    auto normed_product = [&](const float *w, const StepPhase &ph, const Share &one, const float *gain, const float *bias, float *part) {
        float mean[MR], sd[MR];
        Share r = one;
#pragma unroll 1
        for (int item = first; item < ph.groups * ph.splits; item += gridDim.x) {
            if (item != first) {
                r = share_of(ph, item);
                fetch(wv, w, ph, r);
                fetch_norm(r, gain, bias);
                __syncthreads();
            }
            if (warp * 32 < r.rows) {
                row_statistics<MR>(moments, d, mean, sd);
#pragma unroll 1
                for (int k = tid; k < r.rows; k += kThreads) {
                    const float ga = k == tid ? gain0 : __ldg(gain + r.k0 + k), be = k == tid ? bias0 : __ldg(bias + r.k0 + k);
#pragma unroll
                    for (int m = 0; m < MR; ++m) xs[m * widest + k] = (res[m * d + r.k0 + k] - mean[m]) / sd[m] * ga + be;
                }
            }
            __syncthreads();
            item_product<MR>(wv, w, ph, r, xs, widest, red, part);
        }
    };

    fetch_norm(of_qkv, s.ln1_w, s.ln1_b);
    // a head's size is a power of two: lanes of a cached row, rows at a time
    const int head_log = 31 - __clz(s.hd), per_pos = s.hd >> 2, groups = kThreads / per_pos;
    const int g = tid >> (head_log - 2), c4 = (tid & (per_pos - 1)) * 4, row_stride = 2 * d * groups;
    const size_t dd = static_cast<size_t>(d) * d, df = static_cast<size_t>(d) * s.ffn;
    // half layers: qkv, attention, projection; up, GELU, down.  Their common parts are in the code once: inlined per use the kernel had 150 KB of code,
    // more than the instruction caches hold.
#pragma unroll 1
    for (int n = 0;; ++n) {
        const int l = n >> 1;
        const bool half = n & 1;
        if (n > 0) add_result(half ? s.proj_part : s.down_part, half ? s.proj : s.down, half ? s.proj_b + l * d : s.down_b + (l - 1) * d);
        if (n == 2 * s.layers) break;
        normed_product(half ? s.up_w + df * l : s.qkv_w + 3 * dd * l, half ? s.up : s.qkv, half ? of_up : of_qkv, (half ? s.ln2_w : s.ln1_w) + l * d, (half ? s.ln2_b : s.ln1_b) + l * d,
                       half ? s.up_part : s.qkv_part);
        arrive(s, target);
        const float *w = half ? s.down_w + df * l : s.proj_w + dd * l;
        const StepPhase ph = half ? s.down : s.proj;
        const Share mine_of = half ? of_down : of_proj;
        fetch(wv, w, ph, mine_of);
        float *cache = s.cache + static_cast<size_t>(l) * MR * s.max_len * 2 * d;
        // and the first cached rows of this block's first head
        float4 k_first[4], v_first[4];
        {
            const float *row = cache + static_cast<size_t>(g) * 2 * d + of_proj.k0 + c4;
#pragma unroll
            for (int j = 0; j < 4; ++j, row += row_stride) {
                const bool live = !half && of_proj.rows > 0 && g + j * groups < p;
                k_first[j] = live ? *reinterpret_cast<const float4 *>(row) : make_float4(0.f, 0.f, 0.f, 0.f);
                v_first[j] = live ? *reinterpret_cast<const float4 *>(row + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        await(s, target, gave_up);

        Share r = mine_of;
#pragma unroll 1
        for (int item = first; item < ph.groups * ph.splits; item += gridDim.x) {
            if (item != first) {
                r = share_of(ph, item);
                fetch(wv, w, ph, r);
            }
            if (half) {   // the finished up product through the GELU
                if (item != first) __syncthreads();
#pragma unroll 1
                for (int m = 0; m < MR; ++m)
#pragma unroll 1
                    for (int k = tid; k < r.rows; k += kThreads) {
                        const float be = __ldg(s.up_b + l * s.ffn + r.k0 + k);
                        xs[m * widest + k] = gelu_tanh(sum_parts(s.up_part + m * s.ffn + r.k0 + k, s.up.splits, MR * s.ffn) + be);
                    }
            }
            // or the attention of the heads in the item's slice of k
#pragma unroll 1
            for (int at = half ? r.rows : 0; at < r.rows; at += s.hd) {
                const bool fetched = item == first && at == 0;   // k_first, v_first are this head's, row 0
                if (!fetched) __syncthreads();
#pragma unroll 1
                for (int i = tid; i < MR * 3 * s.hd; i += kThreads) {
                    const int row = i >> head_log, m = MR == 1 ? 0 : row / 3, which = row - 3 * m, e = i & (s.hd - 1), col = which * d + r.k0 + at + e;
                    const float be = __ldg(s.qkv_b + l * 3 * d + col);
                    const float v = sum_parts(s.qkv_part + m * 3 * d + col, s.qkv.splits, MR * 3 * d) + be;
                    fresh[i] = v;
                    if (which > 0 && r.col == 0) cache[(static_cast<size_t>(m) * s.max_len + p) * 2 * d + (col - d)] = v;
                }
                __syncthreads();
#pragma unroll 1
                for (int m = 0; m < MR; ++m) {
                    const float *q = fresh + m * 3 * s.hd + c4, *row = cache + (static_cast<size_t>(m) * s.max_len + g) * 2 * d + r.k0 + at + c4;
                    const float4 q4 = *reinterpret_cast<const float4 *>(q);
                    float *probs = prob + m * s.max_len;
#pragma unroll 1
                    for (int t0 = 0; t0 <= p; t0 += 4 * groups, row += 4 * row_stride) {   // four rows in flight per thread
                        float4 kv[4];
                        float v[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int t = t0 + g + j * groups;
                            kv[j] = fetched && m == 0 && t0 == 0 ? k_first[j] : t < p ? *reinterpret_cast<const float4 *>(row + j * row_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
                            if (t == p) kv[j] = *reinterpret_cast<const float4 *>(q + s.hd);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[j] = dot4(q4, kv[j], 0.0f);
#pragma unroll 1
                        for (int o = per_pos >> 1; o > 0; o >>= 1)
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
                        if (c4 == 0)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (t0 + g + j * groups <= p) probs[t0 + g + j * groups] = v[j] * s.scale;
                    }
                }
                __syncthreads();
#pragma unroll 1
                for (int m = 0; m < MR; ++m) {
                    const float *q = fresh + m * 3 * s.hd + c4, *row = cache + (static_cast<size_t>(m) * s.max_len + g) * 2 * d + d + r.k0 + at + c4;
                    float *probs = prob + m * s.max_len;
                    float mx = -FLT_MAX, weights = 0.0f;
#pragma unroll 1
                    for (int t = lane; t <= p; t += 32) mx = fmaxf(mx, probs[t]);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                    for (int t0 = 0; t0 + g <= p; t0 += 4 * groups, row += 4 * row_stride) {
                        float4 kv[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int t = t0 + g + j * groups;
                            kv[j] = fetched && m == 0 && t0 == 0 ? v_first[j] : t < p ? *reinterpret_cast<const float4 *>(row + j * row_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
                            if (t == p) kv[j] = *reinterpret_cast<const float4 *>(q + 2 * s.hd);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (t0 + g + j * groups <= p) {
                                const float e = expf(probs[t0 + g + j * groups] - mx);
                                weights += e;
                                acc.x = fmaf(e, kv[j].x, acc.x);
                                acc.y = fmaf(e, kv[j].y, acc.y);
                                acc.z = fmaf(e, kv[j].z, acc.z);
                                acc.w = fmaf(e, kv[j].w, acc.w);
                            }
                    }
#pragma unroll 1
                    for (int o = per_pos; o < 32; o <<= 1) {
                        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
                        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
                        acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
                        weights += __shfl_xor_sync(0xffffffffu, weights, o);
                    }
                    if (m > 0) __syncthreads();   // the previous row's parts have been added up
                    if (lane < per_pos) *reinterpret_cast<float4 *>(out + warp * (s.hd + 4) + c4) = acc;
                    if (lane == 0) out[warp * (s.hd + 4) + s.hd] = weights;
                    __syncthreads();
                    if (tid < s.hd) {   // heads are at most 128 wide
                        float v = 0.0f, sum = 0.0f;
#pragma unroll
                        for (int j = 0; j < kWarps; ++j) {
                            v += out[j * (s.hd + 4) + tid];
                            sum += out[j * (s.hd + 4) + s.hd];
                        }
                        xs[m * widest + at + tid] = v / sum;
                    }
                }
            }
            __syncthreads();
            item_product<MR>(wv, w, ph, r, xs, widest, red, half ? s.down_part : s.proj_part);
        }
        arrive(s, target);
        if (n + 1 < 2 * s.layers) {
            const int next = (n + 1) >> 1;
            fetch(wv, half ? s.qkv_w + 3 * dd * next : s.up_w + df * next, half ? s.qkv : s.up, half ? of_qkv : of_up);
            fetch_norm(half ? of_qkv : of_up, (half ? s.ln1_w : s.ln2_w) + next * d, (half ? s.ln1_b : s.ln2_b) + next * d);
        }
        await(s, target, gave_up);
    }

    // final norm; logits: a warp per pair of embedding rows
    {
        float mean[MR], sd[MR];
        row_statistics<MR>(moments, d, mean, sd);
#pragma unroll 1
        for (int k = tid; k < d; k += kThreads)
#pragma unroll
            for (int m = 0; m < MR; ++m) xs[m * widest + k] = (res[m * d + k] - mean[m]) / sd[m] * __ldg(s.lnf_w + k) + __ldg(s.lnf_b + k);
    }
    if (__syncthreads_or(gave_up)) return;
#pragma unroll 1
    for (int n = 2 * (blockIdx.x * kWarps + warp); n < s.vocab_p; n += 2 * kWarps * gridDim.x) {
        const float *wa = s.wte + static_cast<size_t>(n) * d, *wb = n + 1 < s.vocab_p ? wa + d : wa;
        float sa[MR] = {}, sb[MR] = {};
#pragma unroll 1
        for (int k0 = lane * 4; k0 < d; k0 += 6 * 128) {
            float4 a[6], b[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const bool live = k0 + j * 128 < d;
                a[j] = live ? __ldcs(reinterpret_cast<const float4 *>(wa + k0 + j * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
                b[j] = live ? __ldcs(reinterpret_cast<const float4 *>(wb + k0 + j * 128)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                if (k0 + j * 128 >= d) break;
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    const float4 x = *reinterpret_cast<const float4 *>(xs + m * widest + k0 + j * 128);
                    sa[m] = dot4(a[j], x, sa[m]);
                    sb[m] = dot4(b[j], x, sb[m]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MR; ++m) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sa[m] += __shfl_xor_sync(0xffffffffu, sa[m], o);
                sb[m] += __shfl_xor_sync(0xffffffffu, sb[m], o);
            }
            if (lane == 0) {
                s.logits[static_cast<size_t>(m) * s.vocab_p + n] = sa[m];
                if (n + 1 < s.vocab_p) s.logits[static_cast<size_t>(m) * s.vocab_p + n + 1] = sb[m];
            }
        }
    }
    if (blockIdx.x == 0 && tid == 0) {   // every block has passed a barrier since it read them
        *s.pos = p + 1;
        s.sync[1] = target;
    }
}

// ---- three to 64 rows --------------------------------------------------------------------------------------------------------
// Here the fp32 FMAs weigh as much as the weights (64 rows: 10.9 GFLOP for the layers of GPT-2 124M, 0.15 ms of all FMA lanes), so an item's
// weights and activations sit in shared memory and a thread computes ROWS / 8 rows x 8 columns, each quarter of the block a quarter of the
// slice's k (reads of 16 bytes bound the loop: 4 x 4 values per thread over all of k took 13200 cycles for an item of 128 x 128, 8 x 4 with
// the activations stored twice 17300, 8 x 8 10700; the FMAs alone 8200).  An item is 128 columns x up to 128 k-rows (64 KB of weights).  The
// next item's weights are requested a piece at a time inside the main loop, into the other buffer: all at once the threads wait for HBM to
// take them (3000 cycles), and as bulk copies one warp needs 6000 cycles to issue 128 rows.  The norms, the attention and the GELU are
// phases of their own: eight barriers per layer.  Every kind of phase is in the code once: inlined per use the kernel had 184 KB of code, more than
// the instruction caches hold, and its norms and staging took twice as long.
// 64 rows at position 64 - 96: 777 us per step and 143 for the un-embedding, against 1450 as 89 launches (of 128 registers, with 132 bytes spilled).  An item of 128 x 128 takes 3400 cycles to stage,
// 12000 to multiply and 2800 to add up and store; a barrier 2400, the attention of 768 heads 24000.
constexpr int kWideCols = 128, kWideSlice = 128;

// x * sigmoid(2 u) = 0.5 x (1 + tanh u) without the cancellation at negative x.
__device__ __forceinline__ float gelu_step(float x)
{
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return __fdividef(x, 1.0f + expf(-2.0f * u));
}

template <int THREADS>
__device__ __forceinline__ void group_sync() { asm volatile("bar.sync %0, %1;" ::"r"(1 + static_cast<int>(threadIdx.x) / THREADS), "n"(THREADS) : "memory"); }

// activations of an item: [k][row], or on the tensor cores [half of k][part][row][64 k] in bf16, 128-byte swizzle
__host__ __device__ constexpr bool wide_tensor(int rows) { return rows >= 16; }
__host__ __device__ constexpr size_t wide_x_floats(int rows) { return wide_tensor(rows) ? size_t(rows) * 192 : size_t(kWideSlice) * (rows + 4); }
__host__ __device__ constexpr size_t wide_shared_floats(int rows) { return size_t(2) * kWideSlice * kWideCols + wide_x_floats(rows) + 256; }   // 1 KB to align
__host__ __device__ constexpr int wide_attention_threads(int rows) { return rows >= 32 ? 64 : 128; }   // per (sequence, head)
// one of the buffers of weights with the activations beside it: what the sums, the norms and the attention use between products (at least)
__host__ __device__ constexpr size_t wide_scratch_floats(int rows) { return size_t(kWideSlice) * kWideCols + size_t(kWideSlice) * (rows + 4); }
// attention: for every item at work a head's new q, k, v, parts of its output and the scores
__host__ __device__ constexpr int wide_attention_floats(int threads, int hd, int max_len) { return 3 * hd + threads / 32 * (hd + 4) + ((max_len + 3) & ~3); }
inline bool wide_attention_fits(int rows, int hd, int max_len)
{
    const int threads = wide_attention_threads(rows);
    return size_t(kThreads / threads) * wide_attention_floats(threads, hd, max_len) <= wide_scratch_floats(rows);
}

template <int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
gpt_step_rows_kernel(const GptStep s)
{
    constexpr int RT = ROWS / 8, P = ROWS + 4;   // rows per thread; pitch of the activations
    extern __shared__ __align__(16) float sm_raw[];
    __shared__ float4 moments[kWarps];
    float *sm = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~uintptr_t(1023));
    float *xs = sm + kWideSlice * kWideCols;      // activations, between two buffers of weights [kWideSlice][kWideCols]
    float *ws = sm, *ws_next = xs + wide_x_floats(ROWS);
    auto scratch = [&] { return ws < xs ? ws : xs; };   // the current buffer of weights and the activations: neighbours, whichever buffer it is
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, d = s.d, batch = s.batch, first = blockIdx.x;
    const int p = *s.pos;
    if (p < 0 || p >= s.max_len || p >= s.max_pos) return;   // all blocks alike
    __shared__ bool gave_up;   // thread 0's; no register is free for it, nor for leaving here
    if (tid == 0) gave_up = lost(s);
    __shared__ __align__(8) unsigned long long step_bar;
    __shared__ uint32_t step_tmem, step_abort;
    uint32_t tmem = 0, bar_phase = 0;
    const uint32_t bar = ptx::smem_u32(&step_bar);
    if constexpr (wide_tensor(ROWS)) {
        if (tid == 0) {
            ptx::mbar_init(bar, 4);
            step_abort = 0u;
            ptx::fence_mbar_init();
        }
        if (warp == 0) {
            ptx::tmem_alloc(ptx::smem_u32(&step_tmem), 512);
            ptx::tmem_relinquish();
        }
        ptx::tc_fence_before();
        __syncthreads();
        ptx::tc_fence_after();
        tmem = ptx::warp_uniform(step_tmem);
    }
    unsigned target = s.sync[1];

    // Piece i of eight of an item's weights into the other buffer: 16 of its k-rows, one per warp; columns beyond the matrix are zeros.
    struct Source {
        const float *at;
        unsigned dst, bytes;
        int rows, stride;
    };
    auto source = [&](const float *w, const StepPhase &ph, int item) {
        const int split = item / ph.groups, col = (item - split * ph.groups) * kWideCols + lane * 4, k0 = split * ph.slice;
        Source r;
        r.rows = item < ph.groups * ph.splits ? min(ph.K - k0, ph.slice) - warp : 0;
        r.bytes = col < ph.N ? 16 : 0;
        r.at = r.bytes ? w + static_cast<size_t>(k0 + warp) * ph.N + col : w;
        r.stride = r.bytes ? kWarps * ph.N : 0;
        r.dst = static_cast<unsigned>(__cvta_generic_to_shared(ws_next + warp * kWideCols + lane * 4));
        return r;
    };
    auto fetch = [&](Source &r) {
        if (r.rows > 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(r.dst), "l"(r.at), "r"(r.bytes) : "memory");
        r.at += r.stride;
        r.dst += kWarps * kWideCols * 4;
        r.rows -= kWarps;
    };
    auto fetch_all = [&](const float *w, const StepPhase &ph, int item) {
        Source r = source(w, ph, item);
#pragma unroll 1
        while (r.rows > 0) fetch(r);
    };

    // The activations of an item, [k][row]: a warp takes pieces of eight rows x sixteen k.
    auto stage = [&](int k0, int rows, const float *x, int pitch) {
        const int pieces = (ROWS / 8) * ((rows + 15) >> 4);
#pragma unroll 1
        for (int t0 = warp; t0 < pieces; t0 += 4 * kWarps) {
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = t0 + i * kWarps, row = (t % (ROWS / 8)) * 8 + (lane & 7), k = (t / (ROWS / 8)) * 16 + (lane >> 3) * 4;
                v[i] = t < pieces && row < batch && k < rows ? __ldcg(reinterpret_cast<const float4 *>(x + static_cast<size_t>(row) * pitch + k0 + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = t0 + i * kWarps, row = (t % (ROWS / 8)) * 8 + (lane & 7), k = (t / (ROWS / 8)) * 16 + (lane >> 3) * 4;
                if (t < pieces && k < rows) {
                    xs[k * P + row] = v[i].x;
                    xs[(k + 1) * P + row] = v[i].y;
                    xs[(k + 2) * P + row] = v[i].z;
                    xs[(k + 3) * P + row] = v[i].w;
                }
            }
        }
    };

    // One phase of products; `next`: where the weights of this block's first item of the next product are.
    const int quarter = warp >> 2, cg = tid & 15, rg = (tid >> 4) & 7;
    constexpr int HT = RT < 4 ? RT : 4, kHalf = HT * 8;   // rows per thread and block in one pass over the sums
    auto product = [&](const float *w, const StepPhase &ph, float *part, const float *x, const float *w_next, const StepPhase &ph_next, int item_next) {
        const int items = ph.groups * ph.splits;
        if (first >= items) fetch_all(w_next, ph_next, item_next);
#pragma unroll 1
        for (int item = first; item < items; item += gridDim.x) {
            const int split = item / ph.groups, col0 = (item - split * ph.groups) * kWideCols, k0 = split * ph.slice, rows = min(ph.K - k0, ph.slice);
            {   // the weights of this item become current
                float *t = ws;
                ws = ws_next;
                ws_next = t;
            }
            stage(k0, rows, x, ph.K);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            const bool last = item + static_cast<int>(gridDim.x) >= items;
            Source coming = source(last ? w_next : w, last ? ph_next : ph, last ? item_next : item + static_cast<int>(gridDim.x));
            unsigned long long acc[RT][4];   // columns (4 cg, + 1), (4 cg + 2, + 3), and the same 64 further on
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = 0ull;
            const int per = (rows + 3) >> 2, kb = quarter * per, ke = min(rows, kb + per);
            const float *wp = ws + kb * kWideCols + cg * 4, *xp = xs + kb * P + rg * RT;
#pragma unroll 1
            for (int k = kb; k < ke; k += 4) {
                fetch(coming);
                // one row per thread: four products meet before the running sum, a quarter as long a chain of roundings (the reads of shared memory bound this
                // form, not its arithmetic)
                unsigned long long four[4] = {};
#pragma unroll
                for (int i = 0; i < 4; ++i, wp += kWideCols, xp += P) {
                    if (k + i >= ke) break;
                    const ulonglong2 wa = *reinterpret_cast<const ulonglong2 *>(wp), wb = *reinterpret_cast<const ulonglong2 *>(wp + 64);
                    float x[RT];
                    if constexpr (RT >= 4) {
#pragma unroll
                        for (int r = 0; r < RT; r += 4) {
                            const float4 v = *reinterpret_cast<const float4 *>(xp + r);
                            x[r] = v.x; x[r + 1] = v.y; x[r + 2] = v.z; x[r + 3] = v.w;
                        }
                    } else {
#pragma unroll
                        for (int r = 0; r < RT; ++r) x[r] = xp[r];
                    }
#pragma unroll
                    for (int r = 0; r < RT; ++r) {
                        const unsigned long long xx = ptx::both(x[r]);
                        auto &sum = RT == 1 ? four : acc[r];
                        sum[0] = ptx::fma2(wa.x, xx, sum[0]);
                        sum[1] = ptx::fma2(wa.y, xx, sum[1]);
                        sum[2] = ptx::fma2(wb.x, xx, sum[2]);
                        sum[3] = ptx::fma2(wb.y, xx, sum[3]);
                    }
                }
                if (RT == 1)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[0][c] = ptx::add2(acc[0][c], four[c]);
            }
#pragma unroll 1
            while (coming.rows > 0) fetch(coming);
            // the quarters' sums meet where this item's weights and activations were
            float *sums = scratch();
#pragma unroll
            for (int h = 0; h < RT; h += HT) {
                __syncthreads();   // the weights and activations, or the sums of the pass before, have been read
#pragma unroll
                for (int r = 0; r < HT; ++r) {
                    float *dst = sums + (quarter * kHalf + rg * HT + r) * kWideCols + cg * 4;
                    *reinterpret_cast<ulonglong2 *>(dst) = make_ulonglong2(acc[h + r][0], acc[h + r][1]);
                    *reinterpret_cast<ulonglong2 *>(dst + 64) = make_ulonglong2(acc[h + r][2], acc[h + r][3]);
                }
                __syncthreads();
#pragma unroll
                for (int i = tid; i < kHalf * (kWideCols / 4); i += kThreads) {
                    const int at = i >> 5, row = at / HT * RT + h + at % HT, c = (i & 31) * 4;
                    if (row >= batch || col0 + c >= ph.N) continue;
                    float4 v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = *reinterpret_cast<const float4 *>(sums + (q * kHalf + at) * kWideCols + c);
                    *reinterpret_cast<float4 *>(part + (static_cast<size_t>(split) * batch + row) * ph.N + col0 + c) = pairwise(v);
                }
            }
            if (!last) __syncthreads();   // the next item's activations go where the sums are
        }
    };

    // The same on the tensor cores, operands in three bf16 parts as in rows_sm100.cuh, a step's products in one accumulator, the leading ones last (TMEM has no room
    // for a second one: their truncation, 2^-23 of a step's sum of 16 k, is the largest error of it).  An item's weights go through registers to TMEM at once (lane = column, 24
    // columns per step of 16 k), four warps issue the products of a step each into an accumulator of its own, and the sixteen warps add up a sixteenth of
    // all accumulators each, in fp32 and in the order of k.
    auto product_tensor = [&](const float *w, const StepPhase &ph, float *part, const float *x, const float *w_next, const StepPhase &ph_next, int item_next) {
        constexpr int kAccs = ROWS == 64 ? 4 : 8, kAccCols = 256 / kAccs, kSlotBase = 256, kMine = ROWS / 4;      // accumulators, split weights behind them, rows per warp
        constexpr uint32_t kIdesc = ptx::make_idesc_bf16(128, ROWS, false, false), kPart = ROWS * 128;
        const int items = ph.groups * ph.splits, set = warp >> 2, q4 = warp & 3, n = q4 * 32 + lane;
        const uint32_t lanes = static_cast<uint32_t>(q4 * 32) << 16, x_at = ptx::smem_u32(xs);
        const ptx::SmemDesc desc_x = ptx::smem_desc_words(x_at, 16, 1024, ptx::kLayoutSw128);
        if (first >= items) fetch_all(w_next, ph_next, item_next);
#pragma unroll 1
        for (int item = first; item < items; item += gridDim.x) {
            const int split = item / ph.groups, col0 = (item - split * ph.groups) * kWideCols, k0 = split * ph.slice, rows = min(ph.K - k0, ph.slice), steps = (rows + 15) >> 4;
            {   // the weights of this item become current
                float *t = ws;
                ws = ws_next;
                ws_next = t;
            }
            // x: pieces of eight k of a row
            constexpr int kUnits = (ROWS * 16 + kThreads - 1) / kThreads;
            float4 v[kUnits][2];
#pragma unroll
            for (int u = 0; u < kUnits; ++u) {
                const int i = tid + u * kThreads, row = i >> 4, k = (i & 15) * 8;
                const float4 *src = reinterpret_cast<const float4 *>(x + static_cast<size_t>(row) * ph.K + k0 + k);
                v[u][0] = row < batch && k < rows ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[u][1] = row < batch && k + 4 < rows ? __ldcg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < kUnits; ++u) {
                const int i = tid + u * kThreads, row = i >> 4, c = i & 15;
                if (row >= ROWS) break;
                const float f[8] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w, v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
                uint32_t p0[4], p1[4], p2[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) rows::split3(f[2 * j], f[2 * j + 1], p0[j], p1[j], p2[j]);
                const uint32_t to = x_at + (c >> 3) * 3 * kPart + row * 128 + (((c & 7) ^ (row & 7)) << 4);
                ptx::sts128(to, p0[0], p0[1], p0[2], p0[3]);
                ptx::sts128(to + kPart, p1[0], p1[1], p1[2], p1[3]);
                ptx::sts128(to + 2 * kPart, p2[0], p2[1], p2[2], p2[3]);
            }
            ptx::fence_proxy_async_smem();
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            const bool last = item + static_cast<int>(gridDim.x) >= items;
            fetch_all(last ? w_next : w, last ? ph_next : ph, last ? item_next : item + static_cast<int>(gridDim.x));
            // weights: sixteen k of a column
#pragma unroll 1
            for (int ks = set; ks < steps; ks += 4) {
                float f[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) f[j] = ks * 16 + j < rows ? ws[(ks * 16 + j) * kWideCols + n] : 0.0f;
                uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) rows::split3(f[2 * j], f[2 * j + 1], p0[j], p1[j], p2[j]);
                const uint32_t slot = tmem + lanes + kSlotBase + ks * kRowsSlotCols;
                rows::tmem_st8(slot, p0);
                rows::tmem_st8(slot + 8, p1);
                rows::tmem_st8(slot + 16, p2);
            }
            rows::tmem_st_wait();
            float acc[kMine];
#pragma unroll
            for (int j = 0; j < kMine; ++j) acc[j] = 0.0f;
#pragma unroll 1
            for (int base = 0; base < steps; base += kAccs) {
                const int count = min(kAccs, steps - base);
                ptx::tc_fence_before();
                __syncthreads();      // the split weights are there; the sums of the steps before have been read
                if (warp < 4) {
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
                        for (int a = warp; a < count; a += 4) {
                            const int ks = base + a;
                            rows::issue_step(tmem + a * kAccCols, tmem + a * kAccCols, tmem + kSlotBase + ks * kRowsSlotCols, desc_x, (ks >> 2) * 3 * kPart + (ks & 3) * 32, kPart, kIdesc);
                        }
                        ptx::mma_commit(bar);
                    }
                    __syncwarp();
                }
                if (!bounded_wait(bar, bar_phase, &step_abort, s.status, DEV_TIMEOUT_EPILOGUE) && tid == 0) {   // as at a barrier that ran out
                    gave_up = true;
                    atomicExch(s.sync + 2, 1u);
                }
                bar_phase ^= 1u;
                __syncwarp();
                ptx::tc_fence_after();
#pragma unroll 1
                for (int a = 0; a < count; ++a) {
                    uint32_t r[kMine];
                    const uint32_t at = tmem + lanes + a * kAccCols + set * kMine;
                    if constexpr (kMine == 4)
                        rows::tmem_ld4(at, r);
                    else
#pragma unroll
                        for (int j = 0; j < kMine; j += 8) rows::tmem_ld8(at + j, r + j);
                    ptx::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < kMine; ++j) acc[j] += __uint_as_float(r[j]);
                }
            }
            if (col0 + n < ph.N) {
#pragma unroll
                for (int j = 0; j < kMine; ++j)
                    if (set * kMine + j < batch) part[(static_cast<size_t>(split) * batch + set * kMine + j) * ph.N + col0 + n] = acc[j];
            }
            ptx::tc_fence_before();
            if (!last) __syncthreads();   // every warp has read its sums: the next item's products may overwrite them
        }
    };

    // act = gelu(finished up product), written over the first slice's sums
    auto gelu_phase = [&](const float *bias) {
        const int quads = s.ffn >> 2;
#pragma unroll 1
        for (int i = first * kThreads + tid; i < batch * quads; i += gridDim.x * kThreads) {
            const int row = i / quads, c = (i - row * quads) * 4;
            const float4 be = __ldg(reinterpret_cast<const float4 *>(bias + c));
            float *at = s.up_part + static_cast<size_t>(row) * s.ffn + c;
            const float4 v = add4(sum_parts4<6>(at, s.up.splits, batch * s.ffn), be);
            *reinterpret_cast<float4 *>(at) = make_float4(gelu_step(v.x), gelu_step(v.y), gelu_step(v.z), gelu_step(v.w));
        }
    };

    // res += a finished product (none: the embedding), normed = its norm; a block per row
    auto norm_phase = [&](const float *part, const StepPhase &ph, const float *bias, const float *gain, const float *shift) {
        float *row_sm = scratch(), *half_sm = row_sm + d;   // both fit: see the plan
        constexpr int kSide = kThreads / 2;
        const int half = tid / kSide, at = (tid % kSide) * 4, cut = (ph.splits + 1) / 2;
        const auto at4 = [](const float *q) { return *reinterpret_cast<const float4 *>(q); };
#pragma unroll 1
        for (int row = first; row < batch; row += gridDim.x) {
            __syncthreads();
            // what does not depend on the sums is on its way before them
            float4 before = make_float4(0.f, 0.f, 0.f, 0.f), more = before, ga = before, be = before;
            if (tid * 4 < d) {
                before = part ? __ldcg(reinterpret_cast<const float4 *>(s.res + row * d + tid * 4)) : at4(s.wte + static_cast<size_t>(s.tokens[row]) * d + tid * 4);
                more = part ? at4(bias + tid * 4) : at4(s.wpe + static_cast<size_t>(p) * d + tid * 4);
                ga = at4(gain + tid * 4);
                be = at4(shift + tid * 4);
            }
            if (part) {   // each half of the block adds up half of the slices
#pragma unroll 1
                for (int c = at; c < d; c += kSide * 4)
                    *reinterpret_cast<float4 *>((half ? half_sm : row_sm) + c) = sum_parts4(part + static_cast<size_t>(half ? cut : 0) * batch * d + row * d + c, half ? ph.splits - cut : cut, batch * d);
                __syncthreads();
            }
#pragma unroll 1
            for (int c = tid * 4; c < d; c += kThreads * 4) {
                if (c != tid * 4) {
                    before = part ? __ldcg(reinterpret_cast<const float4 *>(s.res + row * d + c)) : at4(s.wte + static_cast<size_t>(s.tokens[row]) * d + c);
                    more = part ? at4(bias + c) : at4(s.wpe + static_cast<size_t>(p) * d + c);
                }
                const float4 v = add4(before, part ? add4(add4(at4(row_sm + c), at4(half_sm + c)), more) : more);
                *reinterpret_cast<float4 *>(row_sm + c) = v;
                __stcg(reinterpret_cast<float4 *>(s.res + row * d + c), v);
            }
            warp_moments<1>(row_sm, d, moments);   // a thread reads what it wrote
            __syncthreads();
            if (warp * 128 >= d) continue;
            float mean[1], sd[1];
            row_statistics<1>(moments, d, mean, sd);
#pragma unroll 1
            for (int c = tid * 4; c < d; c += kThreads * 4) {
                if (c != tid * 4) {
                    ga = at4(gain + c);
                    be = at4(shift + c);
                }
                const float4 v = at4(row_sm + c);
                *reinterpret_cast<float4 *>(s.normed + row * d + c) = make_float4((v.x - mean[0]) / sd[0] * ga.x + be.x, (v.y - mean[0]) / sd[0] * ga.y + be.y,
                                                                                  (v.z - mean[0]) / sd[0] * ga.z + be.z, (v.w - mean[0]) / sd[0] * ga.w + be.w);
            }
        }
    };

    constexpr int kAtt = wide_attention_threads(ROWS), kAttItems = kThreads / kAtt, kAttWarps = kAtt / 32;
    const int head_log = 31 - __clz(s.hd), per_pos = s.hd >> 2, groups = kAtt / per_pos;
    const int worker = tid / kAtt, qt = tid & (kAtt - 1), g = qt >> (head_log - 2), c4 = (qt & (per_pos - 1)) * 4, row_stride = 2 * d * groups;
    // The cached rows of this block's items towards L2 while the FMAs of the product before keep HBM idle: 37 MB per layer at 64 sequences of 96.
    auto prefetch_cache = [&](const float *cache) {
        const int lines = (s.hd * 4 + 127) >> 7, per_row = 2 * lines;
#pragma unroll 1
        for (int item = first * kAttItems + worker; item < batch * s.heads; item += gridDim.x * kAttItems) {
            const int m = item / s.heads, at = (item - m * s.heads) << head_log;
            const float *keys = cache + static_cast<size_t>(m) * s.max_len * 2 * d + at;
#pragma unroll 2
            for (int i = qt; i < p * per_row; i += kAtt) {
                const int t = i / per_row, j = i - t * per_row;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(keys + static_cast<size_t>(t) * 2 * d + (j >= lines ? d + (j - lines) * 32 : j * 32)));
            }
        }
    };
    // kAtt threads per (sequence, head); sixteen cached rows in flight per thread, the first keys before the new q, k, v are known, the first
    // values before the softmax
    auto attention = [&](float *cache, const float *qkv_b) {
        constexpr int kFlight = 16;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float *fresh = scratch() + worker * wide_attention_floats(kAtt, s.hd, s.max_len);      // [3][hd]
        float *out = fresh + 3 * s.hd, *prob = out + kAttWarps * (s.hd + 4);                    // [kAttWarps][hd + 4], [max_len]
#pragma unroll 1
        for (int item = first * kAttItems + worker; item < batch * s.heads; item += gridDim.x * kAttItems) {
            const int m = item / s.heads, at = (item - m * s.heads) << head_log;
            float *keys = cache + static_cast<size_t>(m) * s.max_len * 2 * d + at;
            const float *row = keys + static_cast<size_t>(g) * 2 * d + c4;
            float4 kv[kFlight];
            auto load = [&](int t0, const float *src) {
#pragma unroll
                for (int j = 0; j < kFlight; ++j, src += row_stride) kv[j] = t0 + g + j * groups < p ? *reinterpret_cast<const float4 *>(src) : zero;
            };
            load(0, row);
#pragma unroll 1
            for (int i = qt * 4; i < 3 * s.hd; i += kAtt * 4) {
                const int which = i >> head_log, e = i & (s.hd - 1), col = which * d + at + e;
                const float4 be = __ldg(reinterpret_cast<const float4 *>(qkv_b + col));
                const float4 v = add4(sum_parts4<8>(s.qkv_part + static_cast<size_t>(m) * 3 * d + col, s.qkv.splits, batch * 3 * d), be);
                *reinterpret_cast<float4 *>(fresh + i) = v;
                if (which > 0) *reinterpret_cast<float4 *>(keys + static_cast<size_t>(p) * 2 * d + (which - 1) * d + e) = v;
            }
            group_sync<kAtt>();
            const float *q = fresh + c4;
            const float4 q4 = *reinterpret_cast<const float4 *>(q);
#pragma unroll 1
            for (int t0 = 0; t0 <= p; t0 += kFlight * groups) {
                if (t0 > 0) load(t0, row + static_cast<size_t>(t0) * 2 * d);
                float v[kFlight];
#pragma unroll
                for (int j = 0; j < kFlight; ++j) {
                    if (t0 + g + j * groups == p) kv[j] = *reinterpret_cast<const float4 *>(q + s.hd);
                    v[j] = dot4(q4, kv[j], 0.0f);
                }
#pragma unroll 1
                for (int o = per_pos >> 1; o > 0; o >>= 1)
#pragma unroll
                    for (int j = 0; j < kFlight; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
                if (c4 == 0)
#pragma unroll
                    for (int j = 0; j < kFlight; ++j)
                        if (t0 + g + j * groups <= p) prob[t0 + g + j * groups] = v[j] * s.scale;
            }
            load(0, row + d);
            group_sync<kAtt>();
            float mx = -FLT_MAX, weights = 0.0f;
#pragma unroll 2
            for (int t = lane; t <= p; t += 32) mx = fmaxf(mx, prob[t]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            float4 acc = zero;
#pragma unroll 1
            for (int t0 = 0; t0 <= p; t0 += kFlight * groups) {
                if (t0 > 0) load(t0, row + d + static_cast<size_t>(t0) * 2 * d);
#pragma unroll
                for (int j = 0; j < kFlight; ++j) {
                    const int t = t0 + g + j * groups;
                    if (t == p) kv[j] = *reinterpret_cast<const float4 *>(q + 2 * s.hd);
                    if (t <= p) {
                        const float e = expf(prob[t] - mx);
                        weights += e;
                        acc.x = fmaf(e, kv[j].x, acc.x);
                        acc.y = fmaf(e, kv[j].y, acc.y);
                        acc.z = fmaf(e, kv[j].z, acc.z);
                        acc.w = fmaf(e, kv[j].w, acc.w);
                    }
                }
            }
#pragma unroll 1
            for (int o = per_pos; o < 32; o <<= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
                acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
                acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
                weights += __shfl_xor_sync(0xffffffffu, weights, o);
            }
            float *mine = out + (warp & (kAttWarps - 1)) * (s.hd + 4);
            if (lane < per_pos) *reinterpret_cast<float4 *>(mine + c4) = acc;
            if (lane == 0) mine[s.hd] = weights;
            group_sync<kAtt>();
#pragma unroll 1
            for (int i = qt; i < s.hd; i += kAtt) {
                float v = 0.0f, sum = 0.0f;
#pragma unroll
                for (int j = 0; j < kAttWarps; ++j) {
                    v += out[j * (s.hd + 4) + i];
                    sum += out[j * (s.hd + 4) + s.hd];
                }
                s.attn[static_cast<size_t>(m) * d + at + i] = v / sum;
            }
            group_sync<kAtt>();   // the next item writes fresh
        }
    };

    // Four products per layer (qkv, projection, up, down), each behind a phase that makes its input; after the last layer the final norm, and
    // the product with the embedding is another launch.
    fetch_all(s.qkv_w, s.qkv, first);
    const size_t dd = static_cast<size_t>(d) * d, df = static_cast<size_t>(d) * s.ffn;
#pragma unroll 1
    for (int n = 0;; ++n) {
        const int l = n >> 2, kind = n & 3;
        float *cache = s.cache + static_cast<size_t>(l) * batch * s.max_len * 2 * d;
        if ((kind & 1) == 0) {
            const bool attended = kind == 2, end = l == s.layers;
            norm_phase(attended ? s.proj_part : l > 0 ? s.down_part : nullptr, attended ? s.proj : s.down, attended ? s.proj_b + l * d : s.down_b + (l - 1) * d,
                       end ? s.lnf_w : (attended ? s.ln2_w : s.ln1_w) + l * d, end ? s.lnf_b : (attended ? s.ln2_b : s.ln1_b) + l * d);
            if (end) break;
        } else if (kind == 1) {
            attention(cache, s.qkv_b + l * 3 * d);
        } else {
            gelu_phase(s.up_b + l * s.ffn);
        }
        arrive(s, target);
        await(s, target, gave_up);
        if (kind == 0) prefetch_cache(cache);
        const StepPhase ph = kind == 0 ? s.qkv : kind == 1 ? s.proj : kind == 2 ? s.up : s.down, ph_next = kind == 0 ? s.proj : kind == 1 ? s.up : kind == 2 ? s.down : s.qkv;
        const float *w = kind == 0 ? s.qkv_w + 3 * dd * l : kind == 1 ? s.proj_w + dd * l : kind == 2 ? s.up_w + df * l : s.down_w + df * l;
        const float *w_next = kind == 0 ? s.proj_w + dd * l : kind == 1 ? s.up_w + df * l : kind == 2 ? s.down_w + df * l : s.qkv_w + 3 * dd * (l + 1);
        float *part = kind == 0 ? s.qkv_part : kind == 1 ? s.proj_part : kind == 2 ? s.up_part : s.down_part;
        const float *x = kind == 1 ? s.attn : kind == 3 ? s.up_part : s.normed;
        const int item_next = kind == 3 && l + 1 == s.layers ? ph_next.groups * ph_next.splits : first;
        if constexpr (wide_tensor(ROWS))
            product_tensor(w, ph, part, x, w_next, ph_next, item_next);
        else
            product(w, ph, part, x, w_next, ph_next, item_next);
        arrive(s, target);
        await(s, target, gave_up);
    }
    if constexpr (wide_tensor(ROWS)) {
        __syncthreads();
        if (warp == 0) ptx::tmem_dealloc(tmem, 512);
    }
    if (blockIdx.x == 0 && tid == 0 && !gave_up) {   // every block has passed a barrier since it read them
        *s.pos = p + 1;
        s.sync[1] = target;
    }
}

}  // namespace step
}  // namespace gptb200
