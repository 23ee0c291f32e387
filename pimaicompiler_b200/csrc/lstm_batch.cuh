// Interface of the recurrence for many lock-step sequences (lstm_batch.cu).
#pragma once
#include "common.cuh"

namespace pimb200 {

constexpr int kBatchMaxPairs = 74;                      // CTA pairs of a launch
constexpr int kBatchFlagWords = 32;                     // a counter has a 128-byte line
constexpr size_t kBatchFlagBytes = (size_t)kBatchMaxPairs * 2 * kBatchFlagWords * 4;

struct BatchDir {              // one direction of a layer
    const __half* Whh;         // packed [4H, H]
    const float* bias;         // packed [4H]
    const float* G;            // input-projection terms of the launch's steps (fp32)
    const __half* h0;          // [B, H] or NULL
    const __half* c0;          // [B, H] or NULL
    __half* y;
    __half* hn;                // [B, H] or NULL
    __half* cn;
    int reverse;
};
struct BatchArgs {
    BatchDir dir[2];
    int dirs;
    long g_tstride, g_bstride;     // of G, in floats
    // row (t, b) of the output: y + (t / y_fold) * y_tstride + (t % y_fold) * H + b * y_bstride; the exchange goes through it
    long y_tstride, y_bstride;
    int y_fold;
    float* c_state[2];             // [B, H] per direction: cell states between the launches of a sequence
    int H, T, B;
    int begin, steps;              // this launch's share of the T steps, in the order in which they are walked
    uint32_t* counters;            // zeroed ahead of the launch by launch_lstm_batch
    int* status;
    int gen;
    int poll_limit;
    long long* trace;              // optional: 8 clocks per CTA and step of the first trace_ctas CTAs
    int trace_ctas;
};

// Sequences per direction that one launch takes (0: none of this size).
int lstm_batch_capacity(int H, int dirs);
// PIMB200_ERR_UNSUPPORTED when a size or an alignment is not its own.
int launch_lstm_batch(BatchArgs& a, cudaStream_t st);

}  // namespace pimb200
