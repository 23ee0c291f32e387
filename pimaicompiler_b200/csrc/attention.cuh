// Interface of attention.cu.  Both return PIMB200_ERR_UNSUPPORTED for shapes that are not theirs.  row0 (optional, int64 in
// device memory): first row of every sequence in packed keys and values (in the block form queries and outputs too), in
// place of the sequence strides.
#pragma once
#include "common.cuh"

namespace pimb200 {

int launch_attention_decode(const __half* q, const __half* K, const __half* V, const long long* row0, const long long* len_dev, long len_inc,
                            long len_add, long max_len, __half* out, int n_seq, int heads, int head_dim, long kv_stride,
                            long seq_stride, long q_stride, long out_stride, float scale, cudaStream_t st);
int launch_attention_block(const __half* q, const __half* k, const __half* v, const long long* lengths, const long long* row0, __half* out, int n_seq,
                           long max_len, int heads, int head_dim, long row_stride, long seq_stride, long out_row_stride,
                           long out_seq_stride, float scale, cudaStream_t st);

}  // namespace pimb200
