// Planning and launch of the one-launch generation step (gpt_step.cuh).
#include <algorithm>
#include <climits>
#include <cstdint>

#include "ctx_internal.h"
#include "gpt_step.cuh"

namespace gptb200 {
namespace {

constexpr size_t kSharedLimit = 216 * 1024;

// Column groups x slices of k for `blocks` resident blocks.  A block takes its items one after the other (rounds); each costs as long as
// `overhead` k-rows beside its slice, for its inputs and its sums, and every slice is one more partial sum that the next phase reads.  At most
// `longest` rows per slice, a multiple of `quantum`.
StepPhase plan_phase(int K, int N, int blocks, int quantum, int cols, int longest, int most, int overhead)
{
    StepPhase best{};
    long long best_cost = 0;
    const int fewest = (K + longest - 1) / longest;
    for (int splits = fewest; splits <= std::max(most, fewest); ++splits) {
        StepPhase p{K, N, (N + cols - 1) / cols, 0, 0};
        p.slice = ((K + splits - 1) / splits + quantum - 1) / quantum * quantum;
        if (p.slice > longest) continue;
        p.splits = (K + p.slice - 1) / p.slice;
        const long long items = static_cast<long long>(p.groups) * p.splits, rounds = (items + blocks - 1) / blocks;
        const long long cost = rounds * (p.slice + overhead);
        if (!best.splits || cost < best_cost) {
            best_cost = cost;
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

// Shared by both forms: sizes that the kernels take, and whose offsets within a layer's matrix fit an int.
bool plan_shape(GptStep &s)
{
    if (s.batch < 1 || s.batch > kStepMaxBatch || s.layers < 1 || s.max_len < 1) return false;
    if (s.d < 1 || s.ffn < 1 || s.d % 4 || s.ffn % 4 || s.heads < 1 || s.d % s.heads) return false;
    s.hd = s.d / s.heads;
    if (s.hd < 8 || s.hd > 128 || (s.hd & (s.hd - 1))) return false;
    return 3LL * s.d * s.d <= INT_MAX && 1LL * s.d * s.ffn <= INT_MAX;
}

bool plan_small(GptStep &s, int blocks)
{
    if (s.batch > 2) return false;
    constexpr int kAny = 1 << 30, kOverhead = 128;
    s.rows = 0;
    s.qkv = plan_phase(s.d, 3 * s.d, blocks, 32, step::kCols, kAny, 16, kOverhead);
    s.proj = plan_phase(s.d, s.d, blocks, s.hd, step::kCols, kAny, 16, kOverhead);
    s.up = plan_phase(s.d, s.ffn, blocks, 32, step::kCols, kAny, 16, kOverhead);
    s.down = plan_phase(s.ffn, s.d, blocks, 32, step::kCols, kAny, 16, kOverhead);
    const int widest = std::max({s.d, s.qkv.slice, s.proj.slice, s.up.slice, s.down.slice}) + 3;
    return step::small_shared_floats(s.batch, s.d, s.hd, s.max_len, widest) * sizeof(float) <= kSharedLimit;
}

bool plan_rows(GptStep &s, int blocks)
{
    constexpr int kOverhead = 32;
    s.rows = s.batch <= 8 ? 8 : s.batch <= 16 ? 16 : s.batch <= 32 ? 32 : 64;
    s.qkv = plan_phase(s.d, 3 * s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32, kOverhead);
    s.proj = plan_phase(s.d, s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32, kOverhead);
    s.up = plan_phase(s.d, s.ffn, blocks, 8, step::kWideCols, step::kWideSlice, 32, kOverhead);
    s.down = plan_phase(s.ffn, s.d, blocks, 8, step::kWideCols, step::kWideSlice, 32, kOverhead);
    // the norms keep a row and half of its sum there
    return 2 * size_t(s.d) <= step::wide_scratch_floats(s.rows) && step::wide_attention_fits(s.rows, s.hd, s.max_len);
}

size_t scratch_of(const GptStep &s)
{
    return s.batch * (size_t(s.qkv.splits) * 3 * s.d + size_t(s.proj.splits) * s.d + size_t(s.up.splits) * s.ffn + size_t(s.down.splits) * s.d + (s.rows ? 3 * size_t(s.d) : 0));
}

// The operators are not bound to the blocks of option "max_sms".  GPT-2 124M, us per step as one launch on 148 / 128 / 96 / 64 / 32 SMs and operator by
// operator: one sequence 226 / 275 / 289 / 376 / 674 and 379 - 442; eight 493 / 550 / 585 / 682 / 1022 and 566 - 631.
bool plan_forms(const GptStep &shape, int blocks, int num_sms, GptStepForms &f)
{
    f = GptStepForms{shape, shape, false, false};
    if (blocks * 5 < num_sms * 3 || !plan_shape(f.few) || !plan_shape(f.many)) return false;
    f.few_fits = plan_small(f.few, blocks);
    f.many_fits = plan_rows(f.many, blocks);
    return f.few_fits || f.many_fits;
}

}  // namespace

bool gpt_step_enabled(const gptb200_ctx *ctx) { return ctx->skinny && ctx->skinny_rows == 0; }

bool plan_gpt_step(gptb200_ctx *ctx, const GptStep &shape, GptStepForms &f, size_t *scratch_floats)
{
    f = GptStepForms{};
    if (!gpt_step_enabled(ctx) || !plan_forms(shape, step_blocks(ctx), ctx->num_sms, f)) return false;
    *scratch_floats = std::max(f.few_fits ? scratch_of(f.few) : 0, f.many_fits ? scratch_of(f.many) : 0);
    return true;
}

bool gpt_step_replayed(const gptb200_ctx *ctx)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &status) != cudaSuccess) cudaGetLastError();   // the default stream, while another one is captured
    return status == cudaStreamCaptureStatusActive;
}

// All figures: GPT-2's layer counts on 148 SMs, us per step.  The operators come as two figures, replayed from a CUDA graph and called, where the host
// bounds them.
//
// The kernel of one or two rows repeats a head's attention in every column group of the projection, for each sequence and each head of the group's
// slice: `passes` times 0.019 us per layer and position, against 0.043 us for all of them in the other kernel, which takes 14 - 34 us more per layer beside that.
//   width, sequences (passes)  position 96: this / other / operators     480                            1000
//   768, 2 (2)                  306 / 478 / 399, 483                      467 / 664 / 761, 816           720 / 922 / 1687, 1747
//   1024, 2 (4)                 850 / 1212 / 1037, 1137                   1614 / 1596 / 2252, 2365       2532 / 2085 / 3583, 3687
//   1280, 1 (3)                 1249 / 2224 / 1844, 2063                  2113 / 2811 / 3388, 3604       3126 / 3541 / 5342, 5552
//   1280, 2 (6)                 1925 / 2260 / 2019, 2214                  3540 / 2866 / 3474, 3666       5589 / 3606 / 5402, 5609
//   1600, 1 (5)                 2722 / 4219 / 3297, 3541                  4445 / 4991 / 5247, 5498       6735 / 5915 / 7825, 8079
//   1600, 2 (10)                4019 / 4286 / 3480, 3715                  7468 / 4966 / 5330, 5558       -    / 6000 / 7804, 8028
// (The other kernel's figures at 768, and at 1024 at position 96, are those of three rows; 1600 at position 96, and one row at 480, with slightly other slices.)
// The other kernel pads up to four rows to eight, and the operators have kernels for four; their attention is the slower one:
//   768, 3    position 64: 461 / 428, 507    128: 504 / 469, 556    256: 569 / 568, 634    480: 664 / 1065, 1122
//   768, 4                 469 / 434, 507         513 / 478, 556         570 / 711, 763         660 / 1065, 1129
//   1024, 3                1203 / 1035, 1175      1293 / 1445, 1512      1421 / 1817, 1926      1604 / 2307, 2444
//   1600, 3                4165 / 3859, 4071      4380 / 4276, 4436      4648 / 4889, 5060      4991 / 5779, 6003
//   512, 3                 288 / 258, 312         317 / 285, 337         355 / 322, 378         418 / 381, 443
//   768, 8                 477 / 522, 599         534 / 712, 755         589 / 915, 961         693 / 1139, 1201
// and beyond width 1600 their products are long enough to hide the launches (2048, eight layers, position 96, 300, 480):
//   2048, 2 (8 passes)     -                      -                      1117 / 1026, 1066
//   2048, 4                994 / 759, 798         1080 / 990, 1022       1135 / 1116, 1152
//   2048, 8                1124 / 1053, 1101      1223 / 1233, 1280      1283 / 1368, 1415
// From nine rows on both sides run on the tensor cores.  The step's padding and its partial sums grow with the rows, the operators' launches do not: from width 1600
// on they take more than 16 rows (positions 64, 256, 480; operators replayed, called; 1280 beyond 32 rows is left with the step, which they would beat there too):
//   768, 16       446 / 684, 707      580 / 935, 963      698 / 1202, 1191       64      624 / 862, 865      893 / 1190, 1213     1211 / 1564, 1586
//   1024, 16      580 / 797, 822      718 / 1054, 1087    834 / 1331, 1327       64      851 / 1015, 1013    1199 / 1392, 1446    1542 / 1778, 1876
//   1280, 32      860 / 917, 952      1129 / 1226, 1276   1489 / 1583, 1718      64      1262 / 1110, 1128   1902 / 1531, 1702    2534 / 1978, 2322
//   1600, 16      990 / 978, 1022     1143 / 1245, 1300   1301 / 1549, 1581      17      1121 / 1034, 1086   1367 / 1305, 1368    1713 / 1601, 1654
//   1600, 32      1166 / 1100, 1131   1508 / 1431, 1515   1961 / 1805, 2049      64      1717 / 1380, 1395   2468 / 1846, 2058    3174 / 2354, 2576
//   2048, 16 (8)  851 / 820, 863      966 / 1013, 1062    1088 / 1250, 1252      64 (8)  1498 / 1206, 1224   2189 / 1607, 1872    2520 / 2028, 2253
const GptStep *gpt_step_form(const GptStepForms &f, int position, bool replayed)
{
    if (f.few_fits) {
        const int passes = f.few.batch * f.few.proj.slice / f.few.hd;
        if (passes <= 2 || (passes <= 6 && 1LL * (passes - 2) * position * f.few.batch <= 1600)) return &f.few;
        if (!f.many_fits && passes <= 4) return &f.few;
    }
    if (!f.many_fits) return nullptr;
    const int batch = f.many.batch, d = f.many.d;
    if (d >= 1600 && batch > 16) return nullptr;
    if (d > 1600 && position < (batch <= 2 ? 640 : batch <= 4 ? 480 : batch <= 8 ? 256 : 0)) return nullptr;
    if (batch <= 2 && position * 5 < d) return nullptr;
    // a graph is replayed at the positions up to the cache's end
    if (batch <= 4 && replayed && (position + f.many.max_len) / 2 < (d < 768 ? 352 : 160)) return nullptr;
    if (batch <= 4 && d >= 1024 && position < 80) return nullptr;
    return &f.many;
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

int gptb200_plan_generate_step(int num_sms, int batch, int d_model, int d_ffn, int heads, int max_len, int position, int replayed, int *plan10)
{
    using namespace gptb200;
    if (!plan10 || num_sms <= 0) return GPTB200_ERR_INVALID_ARG;
    GptStep shape{};
    shape.batch = batch; shape.layers = 1; shape.d = d_model; shape.ffn = d_ffn; shape.heads = heads; shape.max_len = max_len;
    GptStepForms f;
    const GptStep *s = plan_forms(shape, num_sms, num_sms, f) ? gpt_step_form(f, position, replayed != 0) : nullptr;
    std::fill(plan10, plan10 + 10, 0);
    if (!s) return GPTB200_OK;
    const int out[10] = {s->rows ? 2 : 1, s->rows, s->qkv.splits, s->qkv.slice, s->proj.splits, s->proj.slice, s->up.splits, s->up.slice, s->down.splits, s->down.slice};
    std::copy(out, out + 10, plan10);
    return GPTB200_OK;
}
