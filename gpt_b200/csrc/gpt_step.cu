// Planning and launch of the one-launch generation step (gpt_step.cuh).
#include <algorithm>
#include <cstdint>

#include "ctx_internal.h"
#include "gpt_step.cuh"

namespace gptb200 {
namespace {

constexpr size_t kSharedLimit = 200 * 1024;

// Column groups x slices of k for `blocks` resident blocks: the fewest slices (of a multiple of `quantum` rows) that keep the blocks
// within 3 % as busy as any other number up to 16 does.
StepPhase plan_phase(int K, int N, int blocks, int quantum)
{
    StepPhase best{};
    double best_busy = 0.0;
    for (int splits = 1; splits <= 16; ++splits) {
        StepPhase p{K, N, (N + step::kCols - 1) / step::kCols, 0, 0};
        p.slice = ((K + splits - 1) / splits + quantum - 1) / quantum * quantum;
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

int step_blocks(const gptb200_ctx *ctx) { return ctx->max_sms > 0 ? std::min(ctx->max_sms, ctx->num_sms) : ctx->num_sms; }

}  // namespace

bool gpt_step_enabled(const gptb200_ctx *ctx) { return ctx->skinny && ctx->skinny_rows == 0; }

bool plan_gpt_step(gptb200_ctx *ctx, GptStep &s, size_t *scratch_floats)
{
    if (!gpt_step_enabled(ctx) || s.batch < 1 || s.batch > 2 || s.layers < 1) return false;
    if (s.d % 4 || s.ffn % 4 || s.heads < 1 || s.d % s.heads) return false;
    s.hd = s.d / s.heads;
    if (s.hd < 8 || s.hd > 128 || (s.hd & (s.hd - 1))) return false;
    const int blocks = step_blocks(ctx);
    s.qkv = plan_phase(s.d, 3 * s.d, blocks, 32);
    s.proj = plan_phase(s.d, s.d, blocks, s.hd);
    s.up = plan_phase(s.d, s.ffn, blocks, 32);
    s.down = plan_phase(s.ffn, s.d, blocks, 32);
    if (s.proj.slice > 2 * s.hd) return false;   // every block of a head repeats its attention: few heads per block only
    const int widest = std::max({s.d, s.qkv.slice, s.proj.slice, s.up.slice, s.down.slice}) + 3;
    if (step::small_shared_floats(s.batch, s.d, s.hd, s.max_len, widest) * sizeof(float) > kSharedLimit) return false;
    const size_t b = s.batch;
    *scratch_floats = b * (size_t(s.qkv.splits) * 3 * s.d + size_t(s.proj.splits) * s.d + size_t(s.up.splits) * s.ffn + size_t(s.down.splits) * s.d);
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
    return s.batch == 1 ? launch_small<1>(ctx, s, blocks) : launch_small<2>(ctx, s, blocks);
}

}  // namespace gptb200
