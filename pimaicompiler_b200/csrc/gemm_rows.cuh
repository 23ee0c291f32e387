// Interface of the row-major tcgen05 contraction (gemm_rows.cu) and the host state it shares with gemm_tc.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace pimb200 {
namespace tc {

enum RowsEpilogue { kRowsHalf, kRowsFloat, kRowsArgmax, kRowsCell };

// host state of gemm_tc.cu: tensor-map encoders, the device's status block, the launch generation, the SM count
bool encode_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t row_stride_bytes, uint32_t box_rows,
               int elem_bytes);
bool encode_x_time_major(CUtensorMap* map, const void* base, uint64_t batch, uint64_t steps, uint64_t seq_rows, uint64_t cols,
                         uint64_t ldx_bytes, uint32_t box_t);
bool encode_3d(CUtensorMap* map, const void* base, uint64_t cols, uint64_t batch, uint64_t steps, uint64_t row_stride_bytes,
               uint64_t step_stride_bytes, uint32_t box_b);
int tc_prepare(int* dev, int** status, int* gen);
int tc_sm_count(int dev);

}  // namespace tc

// All return PIMB200_ERR_UNSUPPORTED when the shape or an alignment is not theirs.

// Y[J, N] = act(X W^T + bias) as fp16 or fp32; x_batch > 0: X is batch-first [x_batch][x_seq_rows][K] and the rows of Y are
// numbered time-major (row = t * x_batch + b)
int launch_gemm_rows(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx, int ldy,
                     int act, int y_is_f32, int x_batch, long x_seq_rows, cudaStream_t st, int fixed = 0);

// The largest of fp16(X W^T + bias) of every row in pieces: best_v / best_i [*parts][J], *parts <= gemm_rows_max_parts(N).
int gemm_rows_max_parts(int N);
int launch_gemm_rows_argmax(const __half* W, const __half* X, const __half* bias, float* best_v, int* best_i, int* parts, int N,
                            int K, int J, int ldx, cudaStream_t st);

// One LSTM step of J sequences: gates = X Wx^T + H0 Wh^T + bias (H0 may be NULL), cell update, y = h (+ residual)
struct RowsCell {
    const __half *Wx, *Wh;      // packed [4H, I], [4H, H]
    const float* bias;          // packed [4H]
    const __half* x;
    long x_ld;
    const __half *h0, *c0;      // [J, H] or NULL
    __half* y;
    long y_ld;
    __half *hn, *cn;            // [J, H] or NULL
    const __half* res;
    long res_ld;
    int I, H, J;
};
int launch_gemm_rows_cell(const RowsCell& c, cudaStream_t st);
int launch_lstm_cell_skinny(const RowsCell& c, cudaStream_t st);   // blocks of up to 32 sequences (gemm_skinny.cu)

}  // namespace pimb200
