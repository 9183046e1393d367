// Interface of the one-launch decode step (pi_step.cu) to the engine.
#pragma once
#include "pi_common.cuh"
#include "pi_step_plan.h"

namespace pi {

static constexpr int ST_UP = 4, ST_GATE = 5, ST_DOWN = 6;                                           // places in StepLayer::w (those of the dense ones are the numbers above)
static constexpr int ST_N1W = 0, ST_N1B = 1, ST_N2W = 2, ST_N2B = 3, ST_BQKV = 4, ST_BO = 5, ST_BUP = 6, ST_BDOWN = 7;

// a layer's pointers, as the kernel reads them (n2: the FFN's norm; falcon: attn_norm2)
struct StepLayer { const uint8_t * w[7]; const float * f[8]; uint64_t pad; };

struct StepP {
    const StepLayer * layers; int n_layer;
    int d, F, rank, dq, dkv, n_head, n_head_kv, hd, n_ctx, n_vocab, n_pos, max_batch;
    int q4, falcon, rms, neox, relu, head_type;
    float eps, threshold;
    const __half * tok_embd; const __half * pos_embd; const uint8_t * head; const float * out_w; const float * out_b;
    const float * cs; __half * k_cache; __half * v_cache;
    // words that carry the number of their layer, two of each (by the layer's parity)
    unsigned long long * x, * x2, * qkv, * h, * part; uint32_t * acto, * acts, * hid, * maskw;
    float * pred; int64_t pred_stride; float * logits;
    int32_t * tokens, * positions, * argmax; int fed, token, pos;    // fed: this step's token comes with the launch
    float * logits_host; int32_t * argmax_host;
    long long limit; int look, pad;                                  // cycles of a wait; it looks at the clock where its tries & look == 0
    unsigned int * step_no, * abort, * arrived, * status, * ticket; unsigned long long * best, * rows_total;
    int64_t row_bytes;                                               // of up / gate / down_t
    StepMat mat[ST_N_MAT];
    int slot_bytes, n_slots, window, groups, wpt, off_a, off_b, off_c, off_h, off_part, off_rows;
};

StepDevice step_device();                                             // the current device, as the plan sees it (no device: no SMs)
bool step_fits(const StepPlan & pl, bool q4, bool gated);             // the current context runs all CTAs of the plan at once; readies the kernel for launches
static constexpr int STEP_REFUSED = -1;                               // launch_step: these CTAs cannot run at once on this stream, nothing was launched
int launch_step(const StepP & p, const StepPlan & pl, bool gated, cudaStream_t st);

}  // namespace pi
