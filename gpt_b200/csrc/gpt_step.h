// One generation step of a GPT-2 model (one new token per sequence against the KV cache) as ONE persistent launch: what the
// launcher (gpt_step.cu) and the model driver (gpt_model.cu) share.
#pragma once

#include <cstddef>

struct gptb200_ctx;

namespace gptb200 {

// A product of the step: `groups` of output columns (64 wide in the kernel of one or two rows, 128 in the other) x `splits` slices of k of `slice`
// rows.  The slices' sums meet, neighbours first, where the next phase reads them.
struct StepPhase {
    int K, N, groups, splits, slice;
};

struct GptStep {
    int rows;               // 0: the kernel of one or two rows; else the padded row count of the other
    int batch, layers, d, ffn, heads, hd, vocab_p, max_len, max_pos;
    float scale;
    // weights, fp32; layers of a kind one after another
    const float *wte, *wpe, *ln1_w, *ln1_b, *qkv_w, *qkv_b, *proj_w, *proj_b, *ln2_w, *ln2_b, *up_w, *up_b, *down_w, *down_b, *lnf_w, *lnf_b;
    const int *tokens;      // [batch]
    int *pos;               // position of the new tokens; the step advances it
    float *logits;          // [batch][vocab_p]
    float *cache;           // [layers][batch][max_len][2 d]
    // scratch: partial sums [split][batch][N]; beyond two rows also residual stream, normed rows and attention output [batch][d]
    float *qkv_part, *proj_part, *up_part, *down_part, *res, *normed, *attn;
    StepPhase qkv, proj, up, down;
    unsigned *sync;         // arrivals at the grid barriers so far, arrivals before this launch, whether a wait for them ran out
    int *status;
};

constexpr int kStepMaxBatch = 64;

// A step in both its forms, as far as they fit the model and batch: the kernel of one or two rows, and that of up to 64.
struct GptStepForms {
    GptStep few, many;
    bool few_fits, many_fits;
};

// Plans the forms of a model and batch (whose sizes `shape` holds), and the scratch (floats) that either needs; false: neither fits.
bool plan_gpt_step(gptb200_ctx *ctx, const GptStep &shape, GptStepForms &forms, size_t *scratch_floats);
// The faster one at a position of the text, or over the positions that a captured step is replayed at; null: operator by operator.
const GptStep *gpt_step_form(const GptStepForms &forms, int position, bool replayed);
// Whether the context's stream is being captured into a graph.
bool gpt_step_replayed(const gptb200_ctx *ctx);
// The context's options still ask for the kernels of few rows.
bool gpt_step_enabled(const gptb200_ctx *ctx);
// Launches it; `scratch` as planned, `sync` three words that were zero when the cache was filled.
int run_gpt_step(gptb200_ctx *ctx, GptStep s, float *scratch);

}  // namespace gptb200
