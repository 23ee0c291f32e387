// Interface of the RNN-T greedy loop for many utterances (rnnt_batch.cu).
#pragma once
#include "batch_plan.h"
#include "common.cuh"

namespace pimb200 {

struct GreedyBatchArgs {
    const float* E;            // encoder half of the joint, bias included: utterance u, frame t at E + u * e_utt + t * e_frame
    long e_utt, e_frame;
    int* tokens;               // [n_utts][Tp]
    int* n_tokens;             // [n_utts]
    float* logits;             // optional [n_utts][Tp][V]
    int n_utts, Tp;
    const float* P0;           // [V][4 PH]: layer 0's input terms per label, bias included
    const __half *Whh0, *Wih1, *Whh1;   // packed [4 PH, PH]
    const float* bias1;        // packed [4 PH]
    const __half* W1p;         // [JH, PH]
    const __half* W2;          // [V, JH]
    const float* b2;           // [V]
    int PH, JH, V, blank;
    __half* state;             // hidden states of both layers, exchanged through here (greedy_batch_workspace)
    float* partials;           // partial logits behind them
    uint32_t* counters;
    long long* trace;          // optional: 8 clocks per frame of the first CTA
    int* status;
    int gen;
    int poll_limit;
    // filled in by launch_greedy_batch
    uint32_t* labels;          // (behind the counters)
    int ctas;                  // per group
    int jrows;                 // joint rows per CTA
};

// The plan of a model on the current device (capacity 0: not one of its own), and the bytes behind state / partials / counters.
tc::GreedyPlan greedy_batch_plan(int PH, int JH, int V);
void greedy_batch_workspace(int PH, size_t* state, size_t* partials, size_t* counters);
// PIMB200_ERR_UNSUPPORTED, with nothing launched, where the plan's CTAs are not resident at once
int launch_greedy_batch(GreedyBatchArgs& a, const tc::GreedyPlan& plan, cudaStream_t st);

}  // namespace pimb200
