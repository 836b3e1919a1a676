// Planning and launch of the one-launch generation step (gpt_step.cuh).
#include <algorithm>
#include <cstdint>

#include "ctx_internal.h"
#include "gpt_step.cuh"

namespace gptb200 {
namespace {

constexpr size_t kSharedLimit = 216 * 1024;

// Column groups x slices of k for `blocks` resident blocks: the fewest slices (of a multiple of `quantum` rows) that keep the blocks
// within 3 % as busy as any other number up to `most` does; at most `longest` rows.
StepPhase plan_phase(int K, int N, int blocks, int quantum, int cols, int longest, int most)
{
    StepPhase best{};
    double best_busy = 0.0;
    const int fewest = (K + longest - 1) / longest;
    for (int splits = fewest; splits <= std::max(most, fewest); ++splits) {
        StepPhase p{K, N, (N + cols - 1) / cols, 0, 0};
        p.slice = ((K + splits - 1) / splits + quantum - 1) / quantum * quantum;
        if (p.slice > longest) continue;
        p.splits = (K + p.slice - 1) / p.slice;
        const int items = p.groups * p.splits, rounds = (items + blocks - 1) / blocks;
        const double busy = double(K) / (double(rounds) * p.slice) * p.groups / blocks;   // useful share of the k-rows that all blocks could take
        if (busy > best_busy * 1.03) {
            best_busy = busy;
            best = p;
        }
    }
    return best;
}

template <int MR>
int launch_small(gptb200_ctx *ctx, const GptStep &s, int blocks)
{
    int widest = std::max({s.d, s.qkv.slice, s.proj.slice, s.up.slice, s.down.slice});
    widest = (widest + 3) & ~3;
    const size_t smem = step::small_shared_floats(MR, s.d, s.hd, s.max_len, widest) * sizeof(float);
    const void *kernel = reinterpret_cast<const void *>(step::gpt_step_kernel<MR>);
    if (!ctx->configured.count(kernel)) {
        CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSharedLimit)));
        ctx->configured.insert(kernel);
    }
    void *args[] = {const_cast<GptStep *>(&s), &widest};
    CUDA_TRY(ctx, cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(step::kThreads), args, smem, ctx->stream));
    ctx->launches++;
    return GPTB200_OK;
}

template <int ROWS>
int launch_rows(gptb200_ctx *ctx, const GptStep &s, int blocks)
{
    const void *kernel = reinterpret_cast<const void *>(step::gpt_step_rows_kernel<ROWS>);
    const size_t smem = step::wide_shared_floats(ROWS) * sizeof(float);
    if (!ctx->configured.count(kernel)) {
        CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        ctx->configured.insert(kernel);
    }
    void *args[] = {const_cast<GptStep *>(&s)};
    CUDA_TRY(ctx, cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(step::kThreads), args, smem, ctx->stream));
    ctx->launches++;
    return GPTB200_OK;
}

int step_blocks(const gptb200_ctx *ctx) { return ctx->max_sms > 0 ? std::min(ctx->max_sms, ctx->num_sms) : ctx->num_sms; }

// One or two rows: the blocks of a head repeat its attention and every block norms the whole stream, so few heads per block only.
bool plan_small(GptStep &s, int blocks)
{
    if (s.batch > 2) return false;
    constexpr int kAny = 1 << 30;
    s.rows = 0;
    s.qkv = plan_phase(s.d, 3 * s.d, blocks, 32, step::kCols, kAny, 16);
    s.proj = plan_phase(s.d, s.d, blocks, s.hd, step::kCols, kAny, 16);
    s.up = plan_phase(s.d, s.ffn, blocks, 32, step::kCols, kAny, 16);
    s.down = plan_phase(s.ffn, s.d, blocks, 32, step::kCols, kAny, 16);
    if (s.proj.slice > 2 * s.hd) return false;
    const int widest = std::max({s.d, s.qkv.slice, s.proj.slice, s.up.slice, s.down.slice}) + 3;
    return step::small_shared_floats(s.batch, s.d, s.hd, s.max_len, widest) * sizeof(float) <= kSharedLimit;
}

bool plan_rows(GptStep &s, int blocks)
{
    s.rows = s.batch <= 8 ? 8 : s.batch <= 16 ? 16 : s.batch <= 32 ? 32 : 64;
    s.qkv = plan_phase(s.d, 3 * s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32);
    s.proj = plan_phase(s.d, s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32);
    s.up = plan_phase(s.d, s.ffn, blocks, 8, step::kWideCols, step::kWideSlice, 32);
    s.down = plan_phase(s.ffn, s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32);
    // the norms keep a row and half of its sum there
    return 2 * size_t(s.d) <= step::wide_scratch_floats(s.rows) && step::wide_attention_fits(s.rows, s.hd, s.max_len);
}

}  // namespace

bool gpt_step_enabled(const gptb200_ctx *ctx) { return ctx->skinny && ctx->skinny_rows == 0; }

bool plan_gpt_step(gptb200_ctx *ctx, GptStep &s, size_t *scratch_floats)
{
    if (!gpt_step_enabled(ctx) || s.batch < 1 || s.batch > kStepMaxBatch || s.layers < 1) return false;
    if (s.d % 4 || s.ffn % 4 || s.heads < 1 || s.d % s.heads) return false;
    s.hd = s.d / s.heads;
    if (s.hd < 8 || s.hd > 128 || (s.hd & (s.hd - 1))) return false;
    if (!plan_small(s, step_blocks(ctx)) && !plan_rows(s, step_blocks(ctx))) return false;
    const size_t b = s.batch;
    *scratch_floats = b * (size_t(s.qkv.splits) * 3 * s.d + size_t(s.proj.splits) * s.d + size_t(s.up.splits) * s.ffn + size_t(s.down.splits) * s.d + (s.rows ? 3 * size_t(s.d) : 0));
    return true;
}

int run_gpt_step(gptb200_ctx *ctx, GptStep s, float *scratch)
{
    const size_t b = s.batch;
    auto take = [&](size_t n) { float *at = scratch; scratch += n; return at; };
    s.qkv_part = take(b * s.qkv.splits * 3 * s.d);
    s.proj_part = take(b * s.proj.splits * s.d);
    s.up_part = take(b * s.up.splits * s.ffn);
    s.down_part = take(b * s.down.splits * s.d);
    s.status = ctx->d_status;
    const int blocks = step_blocks(ctx);
    if (!s.rows) return s.batch == 1 ? launch_small<1>(ctx, s, blocks) : launch_small<2>(ctx, s, blocks);
    s.res = take(b * s.d);
    s.normed = take(b * s.d);
    s.attn = take(b * s.d);
    const int rc = s.rows == 8 ? launch_rows<8>(ctx, s, blocks) : s.rows == 16 ? launch_rows<16>(ctx, s, blocks) : s.rows == 32 ? launch_rows<32>(ctx, s, blocks) : launch_rows<64>(ctx, s, blocks);
    return rc ? rc : gptb200_unembed_forward(ctx, s.logits, s.normed, s.wte, s.batch, s.d, s.vocab_p);
}

}  // namespace gptb200

int gptb200_selftest_grid_barrier(gptb200_ctx *ctx, int polls)
{
    using namespace gptb200;
    if (!ctx || polls <= 0 || polls > 100000) return GPTB200_ERR_INVALID_ARG;
    const int rc = ensure_workspace(ctx, 64);
    if (rc) return rc;
    GptStep s{};
    s.sync = reinterpret_cast<unsigned *>(ctx->ws);
    s.status = ctx->d_status;
    CUDA_TRY(ctx, cudaMemsetAsync(s.sync, 0, 3 * sizeof(unsigned), ctx->stream));
    step::barrier_selftest_kernel<<<1, 64, 0, ctx->stream>>>(s, static_cast<unsigned>(polls));
    ctx->launches++;
    CUDA_TRY(ctx, cudaGetLastError());
    return GPTB200_OK;
}
