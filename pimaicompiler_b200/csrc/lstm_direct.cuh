// Interface of the recurrence for few lock-step sequences (lstm_direct.cu).
#pragma once
#include "common.cuh"

namespace pimb200 {

constexpr int kDirectMaxSlots = 16;                      // records per CTA and step: layers x sequences
constexpr int kDirectMaxCtas = 128;                      // H <= 1024, eight hidden units per CTA
constexpr int kDirectSets = 2, kDirectBuffers = 4;
constexpr size_t kDirectSetWords = (size_t)kDirectBuffers * kDirectMaxCtas * kDirectMaxSlots;   // 16-byte records
constexpr size_t kDirectBytes = kDirectSets * kDirectSetWords * 16;

struct DirectArgs {
    const __half* Whh[2];      // packed [4H, H] of layer A and, as a wavefront, layer B
    const __half* WihB;        // packed [4H, H]: layer B's input matrix
    const float* bias[2];
    const float* G;            // layer A's input-projection terms (fp32)
    long g_tstride, g_bstride;
    const __half* h0[2];
    const __half* c0[2];
    __half* y;                 // the last layer's output
    long y_tstride, y_bstride;
    __half* hn[2];
    __half* cn[2];
    uint4* set;                // this launch's four record buffers, all sentinels
    uint4* other_set;          // the next launch's: filled with sentinels by this one
    int* status;
    int gen;
    int H, T, B;
    int reverse;
    int poll_limit;
};

size_t direct_smem(int H, int layers);
// layers 1: up to 16 sequences; layers 2 (a wavefront of two stacked layers): up to 8.  H a multiple of 16 up to 1024.
int launch_lstm_direct(const DirectArgs& a, int layers, cudaStream_t st);

}  // namespace pimb200
