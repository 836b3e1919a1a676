// Recurrences with one decay per head and token (Mamba-2; linear attention with constant decays: steps of one, no skip) over prompts: the
// state-space duality form in chunks of 64 tokens, on tensor cores.
//
// With a_t the running sum of log-decays inside a chunk and S the state before it,
//   y_t = exp(a_t) C_t S + sum_{s <= t} exp(a_t - a_s) dt_s (C_t . B_s) x_s + D x_t
//   S  <- exp(a_end) S + sum_s exp(a_end - a_s) dt_s B_s x_s^T
// One block carries one head's state for 64 of its value columns through the chunks of a request, or of a segment of it, and the next chunk's x, B and C
// arrive while this one is computed.  x, B and C are bf16 as the convolution left them; everything that is fp32 by nature (weights with decays and steps, the
// scaled x, the state) enters a product as the sum of two bf16 values.
//
// Four warps keep the state, 16 value columns each, transposed in fp32 accumulators: as such they are the left operand of y^T = S^T C^T, so that the state never
// passes through shared memory and nothing waits for it.  Four warps compute the weights of the chunk's keys, C . B with decays and steps, for all of them.
// Bound by the state warps' chain of products (two blocks per SM: tensor pipe 38 % busy).  4096 tokens, 64 heads of 64 x 128, us for all launches: 307 with 32
// columns per block, the state handed to output warps as two bf16 terms in shared memory; 264 as now, 191 with sizes known at compile time, 171 with all tokens
// of a chunk at once (the products of eight sums alternate, a state is split once) and the segments' initial states from a launch of their own.  Three prompts of
// 870 tokens, 12 heads of 64 x 64: 43 / 33.
//
// Long requests are cut into segments that run side by side: a first launch computes what each segment alone adds to the state and by
// how much it lets earlier state decay, a second one turns those into the segments' initial states, the third computes the outputs.
#pragma once

#include "mamba2.cuh"

namespace gptb200 {
namespace dec {

constexpr int kChunk = 64;
constexpr int kChunkCols = 64;       // value columns per block
constexpr int kChunkThreads = 256;
constexpr int kChunkMaxState = 128;

namespace mma16 {

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Fragments from a row-major tile in shared memory (pitch in bytes), 16 x 16 at (row, col):
//   a_frag     A operand, M = rows, K = columns
//   a_frag_t   A operand, M = columns, K = rows
//   b_frag     two B operands, N = rows (r[0], r[1]: rows 0-7; r[2], r[3]: rows 8-15), K = columns
//   b_frag_t   two B operands, N = columns (r[0], r[1]: columns 0-7; r[2], r[3]: 8-15), K = rows
__device__ __forceinline__ void a_frag(uint32_t (&r)[4], uint32_t tile, int pitch, int row, int col, int lane)
{
    ldsm4(r, tile + (row + (lane & 15)) * pitch + (col + ((lane >> 4) << 3)) * 2);
}
__device__ __forceinline__ void a_frag_t(uint32_t (&r)[4], uint32_t tile, int pitch, int row, int col, int lane)
{
    ldsm4t(r, tile + (row + (lane & 7) + ((lane >> 4) << 3)) * pitch + (col + (((lane >> 3) & 1) << 3)) * 2);
}
__device__ __forceinline__ void b_frag(uint32_t (&r)[4], uint32_t tile, int pitch, int row, int col, int lane)
{
    ldsm4(r, tile + (row + (lane & 7) + ((lane >> 4) << 3)) * pitch + (col + (((lane >> 3) & 1) << 3)) * 2);
}
__device__ __forceinline__ void b_frag_t(uint32_t (&r)[4], uint32_t tile, int pitch, int row, int col, int lane)
{
    ldsm4t(r, tile + (row + (lane & 15)) * pitch + (col + ((lane >> 4) << 3)) * 2);
}

// Two floats as the sum of two bf16 pairs.
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo)
{
    hi = ptx::pack_bf16x2(a, b);
    lo = ptx::pack_bf16x2(a - bf16_lo(hi), b - bf16_hi(hi));
}

}  // namespace mma16

// 16-wide tiles of the state's rows, a size known at compile time: with run-time bounds every product had a branch around it (2 200 instead of 1 000
// instructions per warp and chunk).  Rows beyond the state are zeros.
__host__ __device__ constexpr int chunk_state_tiles(int state) { return state <= 64 ? 4 : 8; }

__host__ __device__ constexpr int chunk_smem_bytes(int tiles)
{
    const int np = (16 * tiles + 8) * 2, xp = (kChunkCols + 8) * 2, wp = (kChunk + 8) * 2;
    return 2 * kChunk * (2 * np + xp) + 2 * kChunk * wp + 2 * 4 * kChunk * 4;
}

// SEGMENT_STATES: only what a segment adds to the state, from zero, into segment_state [entry][head][segment][state][vdim] and the
// segment's decay into segment_decay [entry][head][segment]; the last segment is left out.  Otherwise outputs and, in the last
// segment, the request's new state.  dt null: steps of one; ld_decay: row pitch of log_decay (0: constant decays); d_skip null: none.
// grid: (heads * column slices, entries, segments)
template <bool SEGMENT_STATES, int NT>
__global__ void __launch_bounds__(kChunkThreads, 2)
mamba_chunk_kernel(float *__restrict__ y, const __nv_bfloat16 *__restrict__ xbc, int ld_xbc, const float *__restrict__ dt, const float *__restrict__ log_decay, int ld_decay,
                   const float *__restrict__ d_skip, const RecurrentShape s, const StepEntry *__restrict__ entries, int segment_tokens, int max_segments, float *__restrict__ segment_state,
                   float *__restrict__ segment_decay)
{
    using namespace mma16;
    extern __shared__ __align__(16) uint8_t chunk_smem[];
    grid_dependency_wait();
    grid_dependency_launch();
    const StepEntry e = entries[blockIdx.y];
    const int segment = blockIdx.z, begin = segment * segment_tokens;
    const bool last_segment = begin + segment_tokens >= e.count;
    if (begin >= e.count || (SEGMENT_STATES && last_segment)) return;
    const int count = min(segment_tokens, e.count - begin), first_row = e.row0 + begin;

    const int slices = (s.vdim + kChunkCols - 1) / kChunkCols;
    const int h = blockIdx.x / slices, p0 = (blockIdx.x % slices) * kChunkCols;
    const int P = s.vdim, N = s.state;
    constexpr int NP = 16 * NT;
    const int g = h / (s.heads / s.groups);
    const int cols = min(kChunkCols, P - p0);
    constexpr int np = (NP + 8) * 2, xp = (kChunkCols + 8) * 2, wp = (kChunk + 8) * 2;   // row pitches in bytes
    const int warp = ptx::warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const bool score_role = !SEGMENT_STATES && warp >= 4;
    const int rw = warp & 3;      // warp within its role
    // shared memory: two buffers of [B | C | x], weights of the keys (two terms), per-token values of two chunks
    // (for states alone: four buffers of [B | x], so that a chunk's copies have three chunks' time)
    constexpr int kBufs = SEGMENT_STATES ? 4 : 2, buf_bytes = kChunk * ((SEGMENT_STATES ? 1 : 2) * np + xp);
    static_assert(kBufs * buf_bytes <= 2 * kChunk * (2 * np + xp) + 2 * kChunk * wp, "shared memory");
    const uint32_t base = ptx::smem_u32(chunk_smem);
    const uint32_t wt = base + kBufs * buf_bytes;
    float *tokens = reinterpret_cast<float *>(chunk_smem + 2 * kChunk * (2 * np + xp) + 2 * kChunk * wp);
    auto tile_b = [&](int b) { return base + b * buf_bytes; };
    auto tile_c = [&](int b) { return base + b * buf_bytes + kChunk * np; };
    auto tile_x = [&](int b) { return base + (b + 1) * buf_bytes - kChunk * xp; };
    // running log2-decay, step, decay since the chunk's start, decay to its end times step
    auto cum = [&](int b) { return tokens + b * 4 * kChunk; };
    auto step = [&](int b) { return tokens + b * 4 * kChunk + kChunk; };
    auto up = [&](int b) { return tokens + b * 4 * kChunk + 2 * kChunk; };
    auto down = [&](int b) { return tokens + b * 4 * kChunk + 3 * kChunk; };

    const long long state_floats = static_cast<long long>(s.heads) * N * P;
    float *state = reinterpret_cast<float *>(e.slot + s.ssm_state) + static_cast<long long>(h) * N * P + p0;
    const float *old_state = state + e.parity * state_floats;
    const long long seg0 = (static_cast<long long>(blockIdx.y) * s.heads + h) * max_segments;
    const bool vec = P % 8 == 0 && N % 8 == 0;    // all column offsets are then multiples of 8
    const bool whole = vec && N == NP && cols == kChunkCols;
    const int off_b = s.inner + g * N, off_c = off_b + s.groups * N;

    // One piece of eight columns of a row: 16-byte asynchronous copy, or plain loads where columns are unaligned or end.
    auto piece = [&](uint32_t dst, const __nv_bfloat16 *src, int have) {
        if (vec && have >= 8) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
        } else {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t a = 2 * i < have ? __bfloat16_as_ushort(src[2 * i]) : 0u, b = 2 * i + 1 < have ? __bfloat16_as_ushort(src[2 * i + 1]) : 0u;
                w[i] = a | b << 16;
            }
            ptx::sts128(dst, w[0], w[1], w[2], w[3]);
        }
    };
    // four threads per token
    auto fetch = [&](int chunk, int b) {
        if (chunk * kChunk >= count) {   // beyond the segment: an empty group, so that waits count alike
            asm volatile("cp.async.commit_group;" ::: "memory");
            return;
        }
        const int t = threadIdx.x >> 2, q0 = threadIdx.x & 3;
        const bool in = chunk * kChunk + t < count;
        const __nv_bfloat16 *row = xbc + static_cast<long long>(first_row + (in ? chunk * kChunk + t : 0)) * ld_xbc;
        if (whole) {   // rows beyond the segment are filled with zeros
            const int bytes = in ? 16 : 0;
            auto copy = [&](uint32_t dst, const __nv_bfloat16 *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory"); };
            const uint32_t to = tile_b(b) + t * np + q0 * 16, x_to = tile_x(b) + t * xp + q0 * 16;
            const __nv_bfloat16 *sb = row + off_b + q0 * 8, *sc = row + off_c + q0 * 8, *sx = row + h * P + p0 + q0 * 8;
#pragma unroll
            for (int i = 0; i < NP / 32; ++i) {
                copy(to + i * 64, sb + i * 32);
                if (!SEGMENT_STATES) copy(to + kChunk * np + i * 64, sc + i * 32);
            }
#pragma unroll
            for (int i = 0; i < kChunkCols / 32; ++i) copy(x_to + i * 64, sx + i * 32);
            asm volatile("cp.async.commit_group;" ::: "memory");
            return;
        }
#pragma unroll 1
        for (int q = q0; q < NP / 8; q += 4) {
            piece(tile_b(b) + t * np + q * 16, row + off_b + q * 8, in ? min(8, N - q * 8) : 0);
            if (!SEGMENT_STATES) piece(tile_c(b) + t * np + q * 16, row + off_c + q * 8, in ? min(8, N - q * 8) : 0);
        }
#pragma unroll 1
        for (int q = q0; q < kChunkCols / 8; q += 4) piece(tile_x(b) + t * xp + q * 16, row + h * P + p0 + q * 8, in ? min(8, cols - q * 8) : 0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // per-token values of a chunk by one warp, two tokens per lane: load early, finish later
    constexpr float kLog2e = 1.4426950408889634f;
    float ld[2], sd[2];
    auto load_tokens = [&](int chunk) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = chunk * kChunk + 2 * lane + i;
            const long long row = first_row + t;
            ld[i] = t < count ? log_decay[row * ld_decay + h] * kLog2e : 0.0f;
            sd[i] = t >= count ? 0.0f : dt ? dt[row * s.heads + h] : 1.0f;
        }
    };
    auto finish_tokens = [&](int b) {
        float sum = ld[0] + ld[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += u;
        }
        const float end = __shfl_sync(0xffffffffu, sum, 31), c1 = sum, c0 = sum - ld[1];
        *reinterpret_cast<float2 *>(cum(b) + 2 * lane) = make_float2(c0, c1);
        *reinterpret_cast<float2 *>(step(b) + 2 * lane) = make_float2(sd[0], sd[1]);
        *reinterpret_cast<float2 *>(up(b) + 2 * lane) = make_float2(exp2f(c0), exp2f(c1));
        *reinterpret_cast<float2 *>(down(b) + 2 * lane) = make_float2(exp2f(end - c0) * sd[0], exp2f(end - c1) * sd[1]);
    };

    const int r = lane >> 2, c2 = (lane & 3) * 2;
    // The state of value columns 16 rw ... of this slice: S[j] are 16 columns (rows of the fragment) by state rows 16 k0 + 8 j ...  Without outputs to compute, all
    // eight warps keep states, half of the state rows each.
    constexpr bool kSplitRegs = !SEGMENT_STATES && NT == 8;
    constexpr int kTiles = SEGMENT_STATES ? NT / 2 : NT;      // of 16 state rows
    constexpr int kBatch = kTiles < 4 ? kTiles : 4;           // tiles whose products alternate: a sum is added to every eight products
    const int k0 = SEGMENT_STATES ? (warp >> 2) * kTiles : 0;
    const bool idle = rw * 16 >= cols;                        // no value columns here
    const int chunks = (count + kChunk - 1) / kChunk;
    auto begin_chunk = [&](int ch) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kBufs - 2) : "memory");
        __syncthreads();   // this chunk's tiles and token values are there, the buffer of the chunk before and the weights are free
        fetch(ch + kBufs - 1, (ch + kBufs - 1) % kBufs);
        if (warp == 4 && ch + 1 < chunks) load_tokens(ch + 1);
    };
#pragma unroll
    for (int i = 0; i < kBufs - 1; ++i) fetch(i, i);
    if (warp == 4) {
        load_tokens(0);
        finish_tokens(0);
    }
    if (score_role) {
        if (kSplitRegs) ptx::reg_dec<96>();
        for (int ch = 0; ch < chunks; ++ch) {
            const int b = ch & 1;
            begin_chunk(ch);
            // 16 rows of the chunk against its keys
            float G[8][4] = {};
#pragma unroll 2
            for (int k = 0; k < NT; ++k) {
                uint32_t a[4], f[4][4];
                a_frag(a, tile_c(b), np, rw * 16, k * 16, lane);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j <= rw) b_frag(f[j], tile_b(b), np, j * 16, k * 16, lane);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j <= rw) {
                        mma(G[2 * j], a, f[j][0], f[j][1]);
                        mma(G[2 * j + 1], a, f[j][2], f[j][3]);
                    }
            }
            // decayed, stepped, causal
            const int ta = rw * 16 + r, tb = ta + 8;
            const float ca = cum(b)[ta], cb = cum(b)[tb];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j > 2 * rw + 1) continue;
                const int key = j * 8 + c2;
                const float2 sk = *reinterpret_cast<const float2 *>(step(b) + key), ck = *reinterpret_cast<const float2 *>(cum(b) + key);
                const float w00 = key <= ta ? G[j][0] * exp2f(ca - ck.x) * sk.x : 0.0f, w01 = key + 1 <= ta ? G[j][1] * exp2f(ca - ck.y) * sk.y : 0.0f;
                const float w10 = key <= tb ? G[j][2] * exp2f(cb - ck.x) * sk.x : 0.0f, w11 = key + 1 <= tb ? G[j][3] * exp2f(cb - ck.y) * sk.y : 0.0f;
                uint32_t hi, lo;
                const uint32_t at = wt + ta * wp + key * 2;
                split2(w00, w01, hi, lo);
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(hi) : "memory");
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + kChunk * wp), "r"(lo) : "memory");
                split2(w10, w11, hi, lo);
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + 8 * wp), "r"(hi) : "memory");
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + (kChunk + 8) * wp), "r"(lo) : "memory");
            }
            asm volatile("bar.arrive 1, %0;" ::"n"(kChunkThreads) : "memory");
            if (warp == 4 && ch + 1 < chunks) finish_tokens(b ^ 1);
        }
        return;
    }
    if (kSplitRegs) ptx::reg_inc<160>();   // 128 x 96 + 128 x 160 = 256 x 128 registers
    float S[2 * kTiles][4] = {};
    float decay_all = 1.0f;
    auto each = [&](auto &&f) {
#pragma unroll
        for (int j = 0; j < 2 * kTiles; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int n = k0 * 16 + j * 8 + c2 + (i & 1), p = rw * 16 + r + (i >> 1) * 8;
                f(S[j][i], n < N && p < cols, n * P + p);
            }
    };
    if (!SEGMENT_STATES) {
        const float *init = segment == 0 ? old_state : segment_state + (seg0 + segment - 1) * N * P + p0;
        each([&](float &v, bool ok, int at) { v = ok ? init[at] : 0.0f; });
    }
    const float skip = d_skip ? d_skip[h] : 0.0f;
    for (int ch = 0; ch < chunks; ++ch) {
        const int b = ch & 1, t0 = ch * kChunk;
        begin_chunk(ch);
        if (!SEGMENT_STATES) {
            float Y[8][4] = {};   // eight tokens each
            // contribution of the state before the chunk
#pragma unroll
            for (int k = 0; k < kTiles; ++k) {
                uint32_t hi[4], lo[4], f[4][4];
#pragma unroll
                for (int t = 0; t < 4; ++t) b_frag(f[t], tile_c(b), np, t * 16, k * 16, lane);
#pragma unroll
                for (int i = 0; i < 4; ++i) split2(S[2 * k + (i >> 1)][2 * (i & 1)], S[2 * k + (i >> 1)][2 * (i & 1) + 1], hi[i], lo[i]);
#pragma unroll
                for (int t = 0; t < 8; ++t) mma(Y[t], hi, f[t >> 1][2 * (t & 1)], f[t >> 1][2 * (t & 1) + 1]);
#pragma unroll
                for (int t = 0; t < 8; ++t) mma(Y[t], lo, f[t >> 1][2 * (t & 1)], f[t >> 1][2 * (t & 1) + 1]);
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float2 u = *reinterpret_cast<const float2 *>(up(b) + t * 8 + c2);
                Y[t][0] *= u.x;
                Y[t][1] *= u.y;
                Y[t][2] *= u.x;
                Y[t][3] *= u.y;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kChunkThreads) : "memory");   // the weights of the keys are there
            if (!idle) {
                // the chunk's own tokens up to each row
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t x[4], f[4][4];
                    a_frag_t(x, tile_x(b), xp, kk * 16, rw * 16, lane);
#pragma unroll
                    for (int term = 0; term < 2; ++term) {
#pragma unroll
                        for (int t = kk; t < 4; ++t) b_frag(f[t], wt + term * kChunk * wp, wp, t * 16, kk * 16, lane);
#pragma unroll
                        for (int t = 2 * kk; t < 8; ++t) mma(Y[t], x, f[t >> 1][2 * (t & 1)], f[t >> 1][2 * (t & 1) + 1]);
                    }
                }
                // rows of the fragment are value columns: a quarter warp writes 32 bytes of a token
                float *dst = y + static_cast<long long>(first_row + t0 + c2) * s.inner + h * P + p0 + rw * 16 + r;
                const int left = count - (t0 + c2), below = cols - (rw * 16 + r);
                const bool all = t0 + kChunk <= count && cols == kChunkCols;
#pragma unroll
                for (int t = 0; t < 8; t += 2) {
                    uint32_t x[4];
                    a_frag_t(x, tile_x(b), xp, t * 8, rw * 16, lane);
#pragma unroll
                    for (int q = t; q < t + 2; ++q) {
                        float v[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t xv = x[2 * (q & 1) + (i >> 1)];
                            v[i] = fmaf(skip, (i & 1) ? bf16_hi(xv) : bf16_lo(xv), Y[q][i]);
                        }
                        float *even = dst, *odd = dst + s.inner;
                        if (all) {
                            even[0] = v[0];
                            odd[0] = v[1];
                            even[8] = v[2];
                            odd[8] = v[3];
                        } else {
                            if (q * 8 < left && 0 < below) even[0] = v[0];
                            if (q * 8 + 1 < left && 0 < below) odd[0] = v[1];
                            if (q * 8 < left && 8 < below) even[8] = v[2];
                            if (q * 8 + 1 < left && 8 < below) odd[8] = v[3];
                        }
                        dst += 8 * s.inner;
                    }
                }
            }
        }
        // the state after the chunk
        const float keep = up(b)[kChunk - 1];
        decay_all *= keep;
#pragma unroll
        for (int j = 0; j < 2 * kTiles; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[j][i] *= keep;
        if (!idle) {
#pragma unroll SEGMENT_STATES ? 4 : 2
            for (int kk = 0; kk < kChunk / 16; ++kk) {
                uint32_t x[4], hi[4], lo[4];
                a_frag_t(x, tile_x(ch % kBufs), xp, kk * 16, rw * 16, lane);
                const float2 d0 = *reinterpret_cast<const float2 *>(down(b) + kk * 16 + c2), d1 = *reinterpret_cast<const float2 *>(down(b) + kk * 16 + 8 + c2);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 d = i < 2 ? d0 : d1;
                    split2(d.x * bf16_lo(x[i]), d.y * bf16_hi(x[i]), hi[i], lo[i]);
                }
#pragma unroll
                for (int k = 0; k < kTiles; k += kBatch) {
                    uint32_t f[kBatch][4];
#pragma unroll
                    for (int j = 0; j < kBatch; ++j) b_frag_t(f[j], tile_b(ch % kBufs), np, kk * 16, (k0 + k + j) * 16, lane);
#pragma unroll
                    for (int term = 0; term < 2; ++term)
#pragma unroll
                        for (int j = 0; j < 2 * kBatch; ++j) mma(S[2 * k + j], term ? lo : hi, f[j >> 1][2 * (j & 1)], f[j >> 1][2 * (j & 1) + 1]);
                }
            }
        }
        if (SEGMENT_STATES && warp == 4 && ch + 1 < chunks) finish_tokens(b ^ 1);
    }
    if (SEGMENT_STATES || last_segment) {
        float *dst = SEGMENT_STATES ? segment_state + (seg0 + segment) * N * P + p0 : state + (e.parity ^ 1) * state_floats;
        each([&](float &v, bool ok, int at) {
            if (ok) dst[at] = v;
        });
        if (SEGMENT_STATES && p0 == 0 && warp == 0 && lane == 0) segment_decay[seg0 + segment] = decay_all;
    }
}

// What the segments add -> the states after them: segment_state[i] <- decay_i * (state before) + segment_state[i].
// grid: (heads * blocks of 256 state values, entries)
__global__ void mamba_segments_kernel(float *__restrict__ segment_state, const float *__restrict__ segment_decay, const RecurrentShape s, const StepEntry *__restrict__ entries,
                                      int segment_tokens, int max_segments)
{
    grid_dependency_wait();
    grid_dependency_launch();
    const int size = s.state * s.vdim, blocks = (size + 255) / 256, h = blockIdx.x / blocks, at = blockIdx.x % blocks * 256 + threadIdx.x;
    if (at >= size) return;
    const StepEntry e = entries[blockIdx.y];
    const long long seg0 = (static_cast<long long>(blockIdx.y) * s.heads + h) * max_segments;
    const int segments = (e.count + segment_tokens - 1) / segment_tokens;
    float v = reinterpret_cast<const float *>(e.slot + s.ssm_state)[(static_cast<long long>(e.parity) * s.heads + h) * size + at];
    for (int i = 0; i + 1 < segments; ++i) {
        float *add = segment_state + (seg0 + i) * size + at;
        v = fmaf(v, segment_decay[seg0 + i], *add);
        *add = v;
    }
}

}  // namespace dec
}  // namespace gptb200
