// Row-wise glue operators of the decode path, fp16 storage / fp32 arithmetic: softmax and log_softmax over the last
// dimension, arg max over the last dimension, layer normalisation over the last dimension, tanh and masked_fill.
//
// They stand where the reference's executors forward to libtorch one tensor op at a time
// (runtime/source/executor/op_executor/aten_ops_executor.cpp: executeAtenSoftmax 3402-3436, executeAtenLogSoftmax
// 2092-2133, executeAtenArgmax 520-547, executeAtenLayerNorm 1898-1942, executeAtenTanh 3555-3568,
// executeAtenMaskedFill 2432-2467).  All are small and latency-bound at decode sizes (a 29..32320-wide logit row, a
// handful of attention scores, a 512-wide model vector): one CTA per row (128 threads, 1024 for rows of 4096 elements
// or more), the row is read with 128-bit loads when its address and length allow, reductions run in fp32 through warp
// shuffles and one shared-memory hop.
#include <math_constants.h>

#include "attention.cuh"
#include "common.cuh"

using namespace pimb200;

namespace {

constexpr int kWideRow = 4096;   // rows at least this long get a 1024-thread CTA

template <int T>
__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();   // red may still be read from the previous reduction
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < T / 32; ++w) r = fmaxf(r, red[w]);
    return r;
}
template <int T>
__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < T / 32; ++w) r += red[w];   // fixed order: the result does not depend on timing
    return r;
}

// element access: VEC = 8 halves per 16-byte load when the row allows it, else scalar
template <int T, bool VEC, typename F>
__device__ __forceinline__ void for_each(const __half* row, long cols, F f) {
    if (VEC) {
        const uint4* r4 = reinterpret_cast<const uint4*>(row);
        for (long c = threadIdx.x; c < (cols >> 3); c += T) {
            float xf[8];
            widen8(r4[c], xf);
#pragma unroll
            for (int j = 0; j < 8; ++j) f(c * 8 + j, xf[j]);
        }
    } else {
        for (long c = threadIdx.x; c < cols; c += T) f(c, __half2float(row[c]));
    }
}

// out[c] = g(c, row[c]) for the whole row; in the vector case eight results leave as one 16-byte store
template <int T, bool VEC, typename G>
__device__ __forceinline__ void map_store(const __half* row, __half* out, long cols, G g) {
    if (VEC) {
        const uint4* r4 = reinterpret_cast<const uint4*>(row);
        uint4* o4 = reinterpret_cast<uint4*>(out);
        for (long c = threadIdx.x; c < (cols >> 3); c += T) {
            float xf[8];
            widen8(r4[c], xf);
            __half2 h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __floats2half2_rn(g(c * 8 + 2 * j, xf[2 * j]), g(c * 8 + 2 * j + 1, xf[2 * j + 1]));
            uint4 pk;
            pk.x = *reinterpret_cast<uint32_t*>(&h[0]);
            pk.y = *reinterpret_cast<uint32_t*>(&h[1]);
            pk.z = *reinterpret_cast<uint32_t*>(&h[2]);
            pk.w = *reinterpret_cast<uint32_t*>(&h[3]);
            o4[c] = pk;
        }
    } else {
        for (long c = threadIdx.x; c < cols; c += T) out[c] = __float2half_rn(g(c, __half2float(row[c])));
    }
}

template <int T, bool VEC, bool LOG>
__global__ void __launch_bounds__(T) softmax_rows_kernel(const __half* __restrict__ x, __half* __restrict__ y,
                                                                   long cols) {
    __shared__ float red[T / 32];
    const __half* row = x + (size_t)blockIdx.x * cols;
    __half* out = y + (size_t)blockIdx.x * cols;
    float m = -CUDART_INF_F;
    for_each<T, VEC>(row, cols, [&](long, float v) { m = fmaxf(m, v); });
    m = block_max<T>(m, red);
    float s = 0.f;
    for_each<T, VEC>(row, cols, [&](long, float v) { s += expf(v - m); });
    s = block_sum<T>(s, red);
    const float inv = 1.0f / s, ls = logf(s);
    map_store<T, VEC>(row, out, cols, [&](long, float v) { return LOG ? (v - m) - ls : expf(v - m) * inv; });
}

template <int T, bool VEC>
__global__ void __launch_bounds__(T) argmax_rows_kernel(const __half* x, long long* __restrict__ idx,
                                                                  long cols) {
    __shared__ float red_v[T / 32];
    __shared__ long long red_i[T / 32];
    pdl_launch_dependents();
    pdl_wait();
    const __half* row = x + (size_t)blockIdx.x * cols;
    float bv = -CUDART_INF_F;
    long long bi = cols;   // lowest index among equal maxima wins, as in at::argmax on a contiguous row
    for_each<T, VEC>(row, cols, [&](long c, float v) {
        if (v > bv || (v == bv && c < bi)) { bv = v; bi = c; }
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const long long oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < T / 32; ++w)
            if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bi)) { bv = red_v[w]; bi = red_i[w]; }
        idx[blockIdx.x] = bi < cols ? bi : 0;   // a row of NaNs / -inf only: index 0
    }
}

// The k largest (or smallest) elements of every row, in order, with their indices: k rounds over the row (it stays in
// L1 / L2), each round the block-wide best element that comes after the previous pick in the total order
// (value, then lower index first), so no set of taken indices has to be kept.  One CTA per row.
template <int T>
__global__ void __launch_bounds__(T) topk_rows_kernel(const __half* __restrict__ x, __half* __restrict__ values,
                                                      long long* __restrict__ idx, long cols, int k, int largest) {
    __shared__ float red_v[T / 32];
    __shared__ long long red_i[T / 32];
    __shared__ float pick_v;
    __shared__ long long pick_i;
    const __half* row = x + (size_t)blockIdx.x * cols;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float sgn = largest ? 1.f : -1.f;          // smallest-first is largest-first of the negated row
    float prev_v = CUDART_INF_F;
    long long prev_i = -1;
    for (int r = 0; r < k; ++r) {
        float bv = -CUDART_INF_F;
        long long bi = cols;
        for (long c = threadIdx.x; c < cols; c += T) {
            const float v = sgn * __half2float(row[c]);
            const bool after_prev = v < prev_v || (v == prev_v && c > prev_i);
            if (after_prev && (v > bv || (v == bv && c < bi))) { bv = v; bi = c; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const long long oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0) { red_v[warp] = bv; red_i[warp] = bi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < T / 32; ++w)
                if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bi)) { bv = red_v[w]; bi = red_i[w]; }
            pick_v = bv;
            pick_i = bi;
            const long long out_i = bi < cols ? bi : 0;          // fewer than k comparable elements (NaNs): index 0
            values[(size_t)blockIdx.x * k + r] = row[out_i];
            idx[(size_t)blockIdx.x * k + r] = out_i;
        }
        __syncthreads();
        prev_v = pick_v;
        prev_i = pick_i;
    }
}

template <int T, bool VEC>
__global__ void __launch_bounds__(T) layer_norm_rows_kernel(const __half* __restrict__ x,
                                                                      const __half* __restrict__ gamma,
                                                                      const __half* __restrict__ beta,
                                                                      __half* __restrict__ y, long cols, float eps) {
    __shared__ float red[T / 32];
    const __half* row = x + (size_t)blockIdx.x * cols;
    __half* out = y + (size_t)blockIdx.x * cols;
    float s = 0.f;
    for_each<T, VEC>(row, cols, [&](long, float v) { s += v; });
    const float mean = block_sum<T>(s, red) / (float)cols;
    float q = 0.f;
    for_each<T, VEC>(row, cols, [&](long, float v) { const float d = v - mean; q += d * d; });
    const float rstd = rsqrtf(block_sum<T>(q, red) / (float)cols + eps);   // biased variance, as at::layer_norm
    map_store<T, VEC>(row, out, cols, [&](long c, float v) {
        float r = (v - mean) * rstd;
        if (gamma) r *= __half2float(gamma[c]);
        if (beta) r += __half2float(beta[c]);
        return r;
    });
}

__global__ void tanh_f16_kernel(const __half* __restrict__ x, __half* __restrict__ y, size_t n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        y[i] = __float2half_rn(tanhf(__half2float(x[i])));
}

__global__ void masked_fill_f16_kernel(const __half* __restrict__ x, const unsigned char* __restrict__ mask, __half value,
                                       __half* __restrict__ y, size_t n, size_t mask_n) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        y[i] = mask[i % mask_n] ? value : x[i];
}

// out[i, :] = table[idx[i], :], rows of row_bytes bytes; an index outside [0, n_table) yields a zero row
__global__ void gather_rows_kernel(const unsigned char* table, const long long* idx,
                                   unsigned char* __restrict__ out, size_t row_bytes, long n_table, int vec16) {
    pdl_launch_dependents();
    pdl_wait();
    const long long r = idx[blockIdx.x];
    const bool ok = r >= 0 && r < n_table;
    const unsigned char* src = table + (size_t)(ok ? r : 0) * row_bytes;
    unsigned char* dst = out + (size_t)blockIdx.x * row_bytes;
    if (vec16) {
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        for (size_t i = threadIdx.x; i < row_bytes / 16; i += blockDim.x)
            reinterpret_cast<uint4*>(dst)[i] = ok ? reinterpret_cast<const uint4*>(src)[i] : zero;
    } else {
        for (size_t i = threadIdx.x; i < row_bytes; i += blockDim.x) dst[i] = ok ? src[i] : (unsigned char)0;
    }
}

// table[idx[i], :] = src[i, :]: the write-side twin of the gather (a KV-cache append at a position that lives on the
// device); an index outside [0, n_table) is skipped
__global__ void scatter_rows_kernel(unsigned char* __restrict__ table, const long long* idx,
                                    const unsigned char* src, size_t row_bytes, long n_table, int vec16) {
    pdl_launch_dependents();
    pdl_wait();
    const long long r = idx[blockIdx.x];
    if (r < 0 || r >= n_table) return;
    unsigned char* dst = table + (size_t)r * row_bytes;
    const unsigned char* s = src + (size_t)blockIdx.x * row_bytes;
    if (vec16) {
        for (size_t i = threadIdx.x; i < row_bytes / 16; i += blockDim.x)
            reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(s)[i];
    } else {
        for (size_t i = threadIdx.x; i < row_bytes; i += blockDim.x) dst[i] = s[i];
    }
}

// Single-query (decode-step) multi-head attention over a key / value cache: one CTA per head,
//     out[h] = softmax(scale * q[h] . K[0..L)[h]^T) . V[0..L)[h],   L = *len_dev + len_add (or len_add when len_dev is NULL).
// Scores live in shared memory (fp32), so L is limited by kAttnMaxLen.  Rows of K / V are kv_stride elements apart.
constexpr int kAttnThreads = 128;
constexpr int kAttnMaxLen = 8192;

__global__ void __launch_bounds__(kAttnThreads) attention_row_kernel(const __half* __restrict__ q, const __half* __restrict__ K,
                                                                     const __half* __restrict__ V, const long long* len_dev,
                                                                     long len_add, long max_len, __half* __restrict__ out,
                                                                     int hd, long kv_stride, float scale) {
    extern __shared__ float sc[];            // [L] scores, then [kAttnThreads / 32][hd] partial outputs
    __shared__ float red[kAttnThreads / 32];
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long L = (len_dev ? (long)*len_dev : 0) + len_add;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    const __half* qh = q + (size_t)h * hd;
    // scores: a warp per cache row, lanes along the head dimension
    for (long t = warp; t < L; t += kAttnThreads / 32) {
        const __half* kr = K + (size_t)t * kv_stride + (size_t)h * hd;
        float a = 0.f;
        for (int j = lane; j < hd; j += 32) a = fmaf(__half2float(qh[j]), __half2float(kr[j]), a);
        a = warp_sum(a);
        if (lane == 0) sc[t] = a * scale;
    }
    __syncthreads();
    float m = -CUDART_INF_F;
    for (long t = threadIdx.x; t < L; t += kAttnThreads) m = fmaxf(m, sc[t]);
    m = block_max<kAttnThreads>(m, red);
    float s = 0.f;
    for (long t = threadIdx.x; t < L; t += kAttnThreads) {
        const float e = expf(sc[t] - m);
        sc[t] = e;
        s += e;
    }
    s = block_sum<kAttnThreads>(s, red);   // ends with a barrier: every sc[t] is final
    const float inv = L > 0 ? 1.0f / s : 0.f;
    // weighted sum: warp w takes rows w, w+4, ...; lanes along the head dimension; partials meet in shared memory
    float* part = sc + max_len;
    for (int j = lane; j < hd; j += 32) {
        float a = 0.f;
        for (long t = warp; t < L; t += kAttnThreads / 32)
            a = fmaf(sc[t], __half2float(V[(size_t)t * kv_stride + (size_t)h * hd + j]), a);
        part[warp * hd + j] = a;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < hd; j += kAttnThreads) {
        float a = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnThreads / 32; ++w) a += part[w * hd + j];
        out[(size_t)h * hd + j] = __float2half_rn(a * inv);
    }
}

// Batched form of attention_row_kernel: blockIdx.y is the sequence; every sequence has its own cache (seq_stride
// elements after the previous one) and its own length (len_dev[seq * len_inc]).
__global__ void __launch_bounds__(kAttnThreads) attention_rows_kernel(const __half* __restrict__ q, const __half* __restrict__ K,
                                                                      const __half* __restrict__ V, const long long* row0,
                                                                      const long long* len_dev,
                                                                      long len_inc, long len_add, long max_len,
                                                                      __half* __restrict__ out, int hd, long kv_stride,
                                                                      long seq_stride, long q_stride, long out_stride,
                                                                      float scale) {
    extern __shared__ float sc[];            // [max_len] scores, then [kAttnThreads / 32][hd] partial outputs
    __shared__ float red[kAttnThreads / 32];
    const int h = blockIdx.x, seq = blockIdx.y, heads = gridDim.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long L = (len_dev ? (long)len_dev[(size_t)seq * len_inc] : 0) + len_add;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    (void)heads;
    const __half* qh = q + (size_t)seq * q_stride + (size_t)h * hd;
    const size_t at0 = (row0 ? (size_t)row0[seq] * kv_stride : (size_t)seq * seq_stride) + (size_t)h * hd;
    const __half *Ks = K + at0, *Vs = V + at0;
    for (long t = warp; t < L; t += kAttnThreads / 32) {
        const __half* kr = Ks + (size_t)t * kv_stride;
        float a = 0.f;
        for (int j = lane; j < hd; j += 32) a = fmaf(__half2float(qh[j]), __half2float(kr[j]), a);
        a = warp_sum(a);
        if (lane == 0) sc[t] = a * scale;
    }
    __syncthreads();
    float m = -CUDART_INF_F;
    for (long t = threadIdx.x; t < L; t += kAttnThreads) m = fmaxf(m, sc[t]);
    m = block_max<kAttnThreads>(m, red);
    float s = 0.f;
    for (long t = threadIdx.x; t < L; t += kAttnThreads) {
        const float e = expf(sc[t] - m);
        sc[t] = e;
        s += e;
    }
    s = block_sum<kAttnThreads>(s, red);   // ends with a barrier: every sc[t] is final
    const float inv = L > 0 ? 1.0f / s : 0.f;
    float* part = sc + max_len;
    for (int j = lane; j < hd; j += 32) {
        float a = 0.f;
        for (long t = warp; t < L; t += kAttnThreads / 32) a = fmaf(sc[t], __half2float(Vs[(size_t)t * kv_stride + j]), a);
        part[warp * hd + j] = a;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < hd; j += kAttnThreads) {
        float a = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnThreads / 32; ++w) a += part[w * hd + j];
        out[(size_t)seq * out_stride + (size_t)h * hd + j] = __float2half_rn(a * inv);
    }
}

// Additive (normalised Bahdanau) attention of a decode step:
//     e[s]   = sum_h v[h] * tanh(keys_proj[s, h] + q[h] + bias[h]),  s < length
//     ctx[h] = sum_s softmax(e)[s] * values[s, h]
// Row s of sentence j lies at j * seq_stride + s * row_stride elements (time-major encoder output: row_stride =
// sentences * H, seq_stride = H).  Two launches, both with far more CTAs than SMs, because one CTA per sentence walks
// its 50 rows one dependent load after the other: (1) a warp per (sentence, source position) computes the score,
// (2) a CTA per (sentence, slice of H) turns the sentence's scores into weights and accumulates its slice of the
// context, eight rows of loads in flight per thread.
constexpr int kAddAttnThreads = 256;
constexpr int kAddAttnSlice = 256;       // context elements per CTA of the second launch (two per thread, 128 threads)

__global__ void __launch_bounds__(kAddAttnThreads) additive_scores_kernel(
    const __half* q, const __half* keys_proj, const long long* lengths,
    const __half* v, const __half* bias, float* __restrict__ scores, int n_seq, long max_len,
    int H, long row_stride, long seq_stride) {
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * (kAddAttnThreads / 32) + warp;     // (sentence, position), position fastest
    if (row >= (long)n_seq * max_len) return;
    const int seq = (int)(row / max_len);
    const long s = row % max_len;
    long L = lengths ? (long)lengths[seq] : max_len;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    if (s >= L) return;
    const __half* kr = keys_proj + (size_t)seq * seq_stride + (size_t)s * row_stride;
    const __half* qr = q + (size_t)seq * H;
    float a = 0.f;
    const bool vec = (H % 8 == 0) && (row_stride % 8 == 0) && (seq_stride % 8 == 0) &&
                     ((reinterpret_cast<uintptr_t>(keys_proj) & 15u) == 0) && ((reinterpret_cast<uintptr_t>(q) & 15u) == 0) &&
                     ((reinterpret_cast<uintptr_t>(v) & 15u) == 0) && (!bias || (reinterpret_cast<uintptr_t>(bias) & 15u) == 0);
    if (vec) {
        for (int c = lane; c < (H >> 3); c += 32) {
            float kf[8], qf[8], vf[8], bf[8];
            widen8(ld_v4(reinterpret_cast<const uint4*>(kr) + c), kf);
            widen8(ld_v4(reinterpret_cast<const uint4*>(qr) + c), qf);
            widen8(ld_v4(reinterpret_cast<const uint4*>(v) + c), vf);
            if (bias) widen8(ld_v4(reinterpret_cast<const uint4*>(bias) + c), bf);
#pragma unroll
            for (int i = 0; i < 8; ++i) a = fmaf(vf[i], tanhf_(kf[i] + (qf[i] + (bias ? bf[i] : 0.f))), a);
        }
    } else {
        for (int h = lane; h < H; h += 32)
            a = fmaf(__half2float(v[h]),
                     tanhf_(__half2float(kr[h]) + (__half2float(qr[h]) + (bias ? __half2float(bias[h]) : 0.f))), a);
    }
    a = warp_sum(a);
    if (lane == 0) scores[row] = a;
}

__global__ void __launch_bounds__(kAddAttnSlice / 2) additive_context_kernel(
    const float* scores, const __half* values, const long long* lengths,
    __half* __restrict__ ctx, long max_len, int H, long row_stride, long seq_stride, long ctx_stride, int copies, long copy_stride) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ float sc[];            // [max_len] softmax weights of this sentence
    __shared__ float red[kAddAttnSlice / 64];
    constexpr int T = kAddAttnSlice / 2;
    const int seq = blockIdx.y;
    long L = lengths ? (long)lengths[seq] : max_len;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    float m = -CUDART_INF_F;
    for (long s = threadIdx.x; s < L; s += T) m = fmaxf(m, scores[(size_t)seq * max_len + s]);
    m = block_max<T>(m, red);
    float sum = 0.f;
    for (long s = threadIdx.x; s < L; s += T) {
        const float e = expf(scores[(size_t)seq * max_len + s] - m);
        sc[s] = e;
        sum += e;
    }
    sum = block_sum<T>(sum, red);             // ends with a barrier: every sc[s] is final
    const float inv = L > 0 ? 1.0f / sum : 0.f;
    const int h = blockIdx.x * kAddAttnSlice + threadIdx.x * 2;
    if (h >= H) return;
    const __half* vals = values + (size_t)seq * seq_stride + h;
    __half* out = ctx + (size_t)seq * ctx_stride + h;
    if (h + 1 < H && (row_stride % 2 == 0) && (seq_stride % 2 == 0) && (ctx_stride % 2 == 0) && (copy_stride % 2 == 0) &&
        ((reinterpret_cast<uintptr_t>(values) & 3u) == 0) && ((reinterpret_cast<uintptr_t>(ctx) & 3u) == 0)) {
        float a0 = 0.f, a1 = 0.f;
        long s = 0;
        for (; s + 8 <= L; s += 8) {
            __half2 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const __half2*>(vals + (size_t)(s + i) * row_stride);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 f = __half22float2(x[i]);
                a0 = fmaf(sc[s + i], f.x, a0);
                a1 = fmaf(sc[s + i], f.y, a1);
            }
        }
        for (; s < L; ++s) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(vals + (size_t)s * row_stride));
            a0 = fmaf(sc[s], f.x, a0);
            a1 = fmaf(sc[s], f.y, a1);
        }
        for (int i = 0; i < copies; ++i) *reinterpret_cast<__half2*>(out + i * copy_stride) = __floats2half2_rn(a0 * inv, a1 * inv);
    } else {
        for (int e = 0; e < 2 && h + e < H; ++e) {
            float a = 0.f;
            for (long s = 0; s < L; ++s) a = fmaf(sc[s], __half2float(vals[(size_t)s * row_stride + e]), a);
            for (int i = 0; i < copies; ++i) out[i * copy_stride + e] = __float2half_rn(a * inv);
        }
    }
}

// Both halves in one launch for rows of 16-byte pieces: a cluster of C CTAs per sentence.  The CTAs share the source
// positions for the scores (a warp per position), exchange the scores through distributed shared memory, and share the
// columns of H for the context.  Keys and values are read once each; MUFU bounds the scores, so four tanh share one
// reciprocal: tanh(x) = 1 - 2 / (1 + e^2x), and with d = 1 + e^2x the four quotients v / d come from 1 / (d0 d1 d2 d3)
// (2x is capped at 20, where tanh is 1 in fp32, so the product stays finite; a NaN stays one): 1.25 MUFU per element instead of 2.
// The first rows of values are loaded before the scores are known.  512 sentences (one CTA each): 22 + 13 us as two
// launches; few sentences take up to eight CTAs each.
constexpr int kBahdanauThreads = 256;
constexpr int kBahdanauAhead = 8;        // value rows in flight per thread

__device__ __forceinline__ float ex2_(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <int C, int PER_SM>
__global__ void __launch_bounds__(kBahdanauThreads, PER_SM) bahdanau_kernel(
    const __half* q, const __half* keys_proj, const __half* values,
    const long long* lengths, const __half* v, const __half* bias, __half* __restrict__ ctx,
    float* __restrict__ scores, long max_len, int H, long row_stride, long seq_stride, long ctx_stride, int copies, long copy_stride) {
    constexpr int WARPS = kBahdanauThreads / 32;
    constexpr float kScale = 2.885390082f;                  // 2 / ln 2: e^2x = 2^(kScale x)
    extern __shared__ float bsm[];
    float* qb = bsm;                                        // [H] kScale * (q + bias)
    float* vs = qb + H;                                     // [H]
    float* red = vs + H;                                    // [8 * threads] partial contexts
    float* sc = red + 8 * kBahdanauThreads;                 // [max_len] scores of the sentence, then weights
    __shared__ float vsum[WARPS];
    if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this CTA has started: waited for below
    pdl_launch_dependents();
    pdl_wait();
    const int rank = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    long Ll = lengths ? (long)lengths[seq] : max_len;
    const int L = (int)(Ll < 0 ? 0 : (Ll > max_len ? max_len : Ll));
    const int n8 = H >> 3, nch = n8 / C, groups = kBahdanauThreads / nch;   // 16-byte pieces per row, of this CTA, rows side by side
    const int ch = tid % nch, grp = tid / nch;
    const __half* vals = values + (size_t)seq * seq_stride + (size_t)(rank * nch + ch) * 8;
    uint4 va[kBahdanauAhead];
#pragma unroll
    for (int i = 0; i < kBahdanauAhead; ++i) {
        const int s = grp + i * groups;
        va[i] = s < L ? ld_v4(vals + (size_t)s * row_stride) : make_uint4(0u, 0u, 0u, 0u);
    }
    float my_v = 0.f;
    for (int h = tid; h < H; h += kBahdanauThreads) {
        qb[h] = kScale * (__half2float(q[(size_t)seq * H + h]) + (bias ? __half2float(bias[h]) : 0.f));
        const float f = __half2float(v[h]);
        vs[h] = f;
        my_v += f;
    }
    my_v = warp_sum(my_v);
    if (lane == 0) vsum[warp] = my_v;
    __syncthreads();
    float vtot = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) vtot += vsum[w];
    // the cluster's other CTAs have started: their shared memory may be written
    if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // ---- scores: warp w of CTA r takes positions r + C * (w + 8 i) ----
    for (int s = rank + C * warp; s < L; s += C * WARPS) {
        const uint4* kr = reinterpret_cast<const uint4*>(keys_proj + (size_t)seq * seq_stride + (size_t)s * row_stride);
        float a = 0.f;
#pragma unroll 4
        for (int c = lane; c < n8; c += 32) {
            float k[8];
            widen8(ld_v4(kr + c), k);
#pragma unroll
            for (int o = 0; o < 8; o += 4) {
                const float4 b = *reinterpret_cast<const float4*>(qb + c * 8 + o), w = *reinterpret_cast<const float4*>(vs + c * 8 + o);
                const float d0 = 1.f + ex2_(min_nan(fmaf(k[o], kScale, b.x), 28.85390082f)), d1 = 1.f + ex2_(min_nan(fmaf(k[o + 1], kScale, b.y), 28.85390082f)),
                            d2 = 1.f + ex2_(min_nan(fmaf(k[o + 2], kScale, b.z), 28.85390082f)), d3 = 1.f + ex2_(min_nan(fmaf(k[o + 3], kScale, b.w), 28.85390082f));
                const float p01 = d0 * d1, p23 = d2 * d3;
                const float n01 = fmaf(w.x, d1, w.y * d0), n23 = fmaf(w.z, d3, w.w * d2);
                a = fmaf(fmaf(n01, p23, n23 * p01), rcp_approx(p01 * p23), a);
            }
        }
        a = vtot - 2.f * warp_sum(a);
        if (lane == 0) scores[(size_t)seq * max_len + s] = a;
        if (C == 1) {
            if (lane == 0) sc[s] = a;
        } else if (lane < C) {
            uint32_t dst;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"((uint32_t)__cvta_generic_to_shared(sc + s)), "r"(lane));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(a) : "memory");
        }
    }
    if (C == 1) __syncthreads();
    else {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    // ---- softmax: every warp on its own, then the weights once ----
    float m = -CUDART_INF_F;
    for (int s = lane; s < L; s += 32) m = fmaxf(m, sc[s]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float sum = 0.f;
    for (int s = lane; s < L; s += 32) sum += expf(sc[s] - m);
    sum = warp_sum(sum);
    const float inv = L > 0 ? 1.0f / sum : 0.f;
    // ---- context: this CTA's columns ----
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int s0 = grp; s0 < L; s0 += groups * kBahdanauAhead) {
#pragma unroll
        for (int i = 0; i < kBahdanauAhead; ++i) {
            const int s = s0 + i * groups;
            const float p = s < L ? expf(sc[s] - m) : 0.f;
            float f[8];
            widen8(va[i], f);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = fmaf(p, f[e], acc[e]);
        }
#pragma unroll
        for (int i = 0; i < kBahdanauAhead; ++i) {
            const int s = s0 + (i + kBahdanauAhead) * groups;
            va[i] = s < L ? ld_v4(vals + (size_t)s * row_stride) : make_uint4(0u, 0u, 0u, 0u);   // (0 x inf is a NaN)
        }
    }
    if (groups > 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) red[e * kBahdanauThreads + tid] = acc[e];
        __syncthreads();
        if (grp > 0) return;
        for (int g2 = 1; g2 < groups; ++g2)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] += red[e * kBahdanauThreads + g2 * nch + ch];
    }
    __half2 o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = __floats2half2_rn(acc[2 * e] * inv, acc[2 * e + 1] * inv);
    __half* dst = ctx + (size_t)seq * ctx_stride + (size_t)(rank * nch + ch) * 8;
    for (int i = 0; i < copies; ++i) *reinterpret_cast<uint4*>(dst + i * copy_stride) = *reinterpret_cast<uint4*>(o);
}

// y = layer_norm(x + r) per row: the residual connection and the normalisation behind every Transformer sub-layer in one
// pass (the sum lives in shared memory as fp32; each thread re-reads only the entries it wrote).
template <int T>
__global__ void __launch_bounds__(T) add_layer_norm_rows_kernel(const __half* __restrict__ x, const __half* __restrict__ r,
                                                                const __half* __restrict__ gamma, const __half* __restrict__ beta,
                                                                __half* __restrict__ y, long cols, float eps) {
    extern __shared__ float sum_row[];
    __shared__ float red[T / 32];
    const __half* xr = x + (size_t)blockIdx.x * cols;
    const __half* rr = r + (size_t)blockIdx.x * cols;
    __half* out = y + (size_t)blockIdx.x * cols;
    float s = 0.f;
    for (long c = threadIdx.x; c < cols; c += T) {
        const float v = __half2float(xr[c]) + __half2float(rr[c]);
        sum_row[c] = v;
        s += v;
    }
    const float mean = block_sum<T>(s, red) / (float)cols;
    float q = 0.f;
    for (long c = threadIdx.x; c < cols; c += T) { const float d = sum_row[c] - mean; q += d * d; }
    const float rstd = rsqrtf(block_sum<T>(q, red) / (float)cols + eps);
    for (long c = threadIdx.x; c < cols; c += T) {
        float v = (sum_row[c] - mean) * rstd;
        if (gamma) v *= __half2float(gamma[c]);
        if (beta) v += __half2float(beta[c]);
        out[c] = __float2half_rn(v);
    }
}

// The same for rows of up to 2048 elements, a multiple of 8, 16-byte aligned: a warp per row, the row in registers (NV
// 16-byte pieces per lane), no shared memory and no block-wide barrier.  Many rows: bound by HBM (131072 rows of 512: 155 us
// with a CTA per row, 4 passes of 2-byte accesses); few rows: by latency, so one warp per CTA.
template <int NV>
__global__ void __launch_bounds__(256) add_layer_norm_warp_kernel(const __half* x, const __half* r,
                                                                  const __half* gamma, const __half* beta,
                                                                  __half* __restrict__ y, long rows, int cols, float eps) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * cols);
    const uint4* rr = reinterpret_cast<const uint4*>(r + row * cols);
    const int n8 = cols >> 3;
    float v[NV][8], s = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = lane + 32 * i;
        if (c < n8) {
            float b[8];
            widen8(xr[c], v[i]);
            widen8(rr[c], b);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                v[i][e] += b[e];
                s += v[i][e];
            }
        }
    }
    const float mean = warp_sum(s) / (float)cols;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        if (lane + 32 * i < n8)
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                v[i][e] -= mean;
                q = fmaf(v[i][e], v[i][e], q);
            }
    const float rstd = rsqrtf(warp_sum(q) / (float)cols + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = lane + 32 * i;
        if (c >= n8) continue;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[i][e] *= rstd;
            if (gamma) v[i][e] *= __half2float(gamma[c * 8 + e]);
            if (beta) v[i][e] += __half2float(beta[c * 8 + e]);
        }
        __half2 h[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2half2_rn(v[i][2 * e], v[i][2 * e + 1]);
        reinterpret_cast<uint4*>(y + row * cols)[c] = *reinterpret_cast<uint4*>(h);
    }
}

// Multi-head self-attention over every position of a batch of padded sequences (the encoder side of a Transformer):
// one CTA per (head, sequence) holds the sequence's keys and values of that head in shared memory; a warp per query row
// computes its scores (lanes along the keys), the softmax over the sequence's own length, and the weighted sum (lanes
// along the head dimension).  Query rows past the length give zeros.
constexpr int kBlockAttnThreads = 128;

__global__ void __launch_bounds__(kBlockAttnThreads) attention_block_kernel(
    const __half* __restrict__ Q, const __half* __restrict__ K, const __half* __restrict__ V,
    const long long* __restrict__ lengths, const long long* __restrict__ row0, __half* __restrict__ out, long max_len, int hd,
    long row_stride, long seq_stride, long out_row_stride, long out_seq_stride, float scale) {
    extern __shared__ __align__(16) unsigned char blk_smem[];
    const int h = blockIdx.x, seq = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kp = hd + 2;                                   // padded key row (halves): lanes on different rows, different banks
    __half* Ks = reinterpret_cast<__half*>(blk_smem);         // [max_len][kp]
    __half* Vs = Ks + (size_t)max_len * kp;                   // [max_len][hd]
    float* qs = reinterpret_cast<float*>(Vs + (size_t)max_len * hd);   // [warps][hd]
    float* ps = qs + (kBlockAttnThreads / 32) * hd;           // [warps][max_len]
    long L = lengths ? (long)lengths[seq] : max_len;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    const size_t base = (row0 ? (size_t)row0[seq] * row_stride : (size_t)seq * seq_stride) + (size_t)h * hd;
    const size_t out0 = (row0 ? (size_t)row0[seq] * out_row_stride : (size_t)seq * out_seq_stride) + (size_t)h * hd;
    const long n_rows = row0 ? L : max_len;                   // packed rows: there are none past the length
    for (long i = threadIdx.x; i < L * hd; i += kBlockAttnThreads) {
        const long s_ = i / hd;
        const int c = (int)(i % hd);
        Ks[s_ * kp + c] = K[base + (size_t)s_ * row_stride + c];
        Vs[s_ * hd + c] = V[base + (size_t)s_ * row_stride + c];
    }
    __syncthreads();
    float* qw = qs + warp * hd;
    float* pw = ps + (size_t)warp * max_len;
    for (long qi = warp; qi < n_rows; qi += kBlockAttnThreads / 32) {
        __half* o = out + out0 + (size_t)qi * out_row_stride;
        if (qi >= L) {
            for (int c = lane; c < hd; c += 32) o[c] = __float2half_rn(0.f);
            continue;
        }
        for (int c = lane; c < hd; c += 32) qw[c] = __half2float(Q[base + (size_t)qi * row_stride + c]) * scale;
        __syncwarp();
        float m = -CUDART_INF_F;
        for (long s_ = lane; s_ < L; s_ += 32) {
            float a = 0.f;
            for (int c = 0; c < hd; ++c) a = fmaf(qw[c], __half2float(Ks[s_ * kp + c]), a);
            pw[s_] = a;
            m = fmaxf(m, a);
        }
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o2));
        float sum = 0.f;
        for (long s_ = lane; s_ < L; s_ += 32) {
            const float e = expf(pw[s_] - m);
            pw[s_] = e;
            sum += e;
        }
        sum = warp_sum(sum);
        __syncwarp();
        const float inv = 1.0f / sum;
        for (int c = lane; c < hd; c += 32) {
            float a = 0.f;
            for (long s_ = 0; s_ < L; ++s_) a = fmaf(pw[s_], __half2float(Vs[s_ * hd + c]), a);
            o[c] = __float2half_rn(a * inv);
        }
        __syncwarp();
    }
}

inline unsigned flat_grid(size_t n) {
    const size_t g = (n + 255) / 256;
    return (unsigned)(g > (size_t)kNumSmB200 * 8 ? (size_t)kNumSmB200 * 8 : (g ? g : 1));
}
inline bool rows_ok(long rows, long cols) { return rows > 0 && cols > 0 && rows <= 0x7fffffffL; }

}  // namespace

extern "C" int pimb200_softmax_rows(const void* x, void* y, long rows, long cols, int log_softmax, void* stream) {
    if (rows == 0 || cols == 0) return PIMB200_OK;   // empty tensors carry no storage
    if (!x || !y || !rows_ok(rows, cols)) return PIMB200_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __half* xp = static_cast<const __half*>(x);
    __half* yp = static_cast<__half*>(y);
    const bool vec = cols % 8 == 0 && aligned16(x) && aligned16(y);
    const unsigned grid = (unsigned)rows;
    if (cols >= kWideRow) {
        if (vec) {
            if (log_softmax) softmax_rows_kernel<1024, true, true><<<grid, 1024, 0, st>>>(xp, yp, cols);
            else softmax_rows_kernel<1024, true, false><<<grid, 1024, 0, st>>>(xp, yp, cols);
        } else {
            if (log_softmax) softmax_rows_kernel<1024, false, true><<<grid, 1024, 0, st>>>(xp, yp, cols);
            else softmax_rows_kernel<1024, false, false><<<grid, 1024, 0, st>>>(xp, yp, cols);
        }
    } else if (vec) {
        if (log_softmax) softmax_rows_kernel<128, true, true><<<grid, 128, 0, st>>>(xp, yp, cols);
        else softmax_rows_kernel<128, true, false><<<grid, 128, 0, st>>>(xp, yp, cols);
    } else {
        if (log_softmax) softmax_rows_kernel<128, false, true><<<grid, 128, 0, st>>>(xp, yp, cols);
        else softmax_rows_kernel<128, false, false><<<grid, 128, 0, st>>>(xp, yp, cols);
    }
    return launch_status();
}

extern "C" int pimb200_argmax_rows(const void* x, long long* idx, long rows, long cols, void* stream) {
    if (rows == 0) return PIMB200_OK;
    if (!x || !idx || !rows_ok(rows, cols)) return PIMB200_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __half* xp = static_cast<const __half*>(x);
    const bool vec = cols % 8 == 0 && aligned16(x);
    const unsigned grid = (unsigned)rows;
    auto run = [&](auto kernel, int threads) { return cuda_status(launch_pdl(kernel, dim3(grid), dim3(threads), 0, st, xp, idx, cols)); };
    if (cols >= kWideRow) return vec ? run(argmax_rows_kernel<1024, true>, 1024) : run(argmax_rows_kernel<1024, false>, 1024);
    return vec ? run(argmax_rows_kernel<128, true>, 128) : run(argmax_rows_kernel<128, false>, 128);
}

extern "C" int pimb200_layer_norm_rows(const void* x, const void* gamma, const void* beta, void* y, long rows, long cols,
                                       float eps, void* stream) {
    if (rows == 0 || cols == 0) return PIMB200_OK;
    if (!x || !y || !rows_ok(rows, cols)) return PIMB200_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __half* xp = static_cast<const __half*>(x);
    const __half* g = static_cast<const __half*>(gamma);
    const __half* b = static_cast<const __half*>(beta);
    __half* yp = static_cast<__half*>(y);
    const bool vec = cols % 8 == 0 && aligned16(x) && aligned16(y);
    const unsigned grid = (unsigned)rows;
    if (cols >= kWideRow) {
        if (vec) layer_norm_rows_kernel<1024, true><<<grid, 1024, 0, st>>>(xp, g, b, yp, cols, eps);
        else layer_norm_rows_kernel<1024, false><<<grid, 1024, 0, st>>>(xp, g, b, yp, cols, eps);
    } else {
        if (vec) layer_norm_rows_kernel<128, true><<<grid, 128, 0, st>>>(xp, g, b, yp, cols, eps);
        else layer_norm_rows_kernel<128, false><<<grid, 128, 0, st>>>(xp, g, b, yp, cols, eps);
    }
    return launch_status();
}

extern "C" int pimb200_tanh_f16(const void* x, void* y, size_t n, void* stream) {
    if (n == 0) return PIMB200_OK;
    if (!x || !y) return PIMB200_ERR_BAD_ARG;
    tanh_f16_kernel<<<flat_grid(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __half*>(x),
                                                                                 static_cast<__half*>(y), n);
    return launch_status();
}

extern "C" int pimb200_masked_fill_f16(const void* x, const unsigned char* mask, float value, void* y, size_t n,
                                       size_t mask_n, void* stream) {
    if (n == 0) return PIMB200_OK;
    if (!x || !y || !mask) return PIMB200_ERR_BAD_ARG;
    if (mask_n == 0 || n % mask_n != 0) return PIMB200_ERR_BAD_ARG;
    masked_fill_f16_kernel<<<flat_grid(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(x), mask, __float2half_rn(value), static_cast<__half*>(y), n, mask_n);
    return launch_status();
}

extern "C" int pimb200_gather_rows(const void* table, const long long* idx, void* out, long n_idx, size_t row_bytes,
                                   long n_table, void* stream) {
    if (n_idx == 0 || row_bytes == 0) return PIMB200_OK;
    if (!table || !idx || !out || n_idx < 0 || n_idx > 0x7fffffffL || n_table <= 0) return PIMB200_ERR_BAD_ARG;
    const int vec16 = (row_bytes % 16 == 0 && aligned16(table) && aligned16(out)) ? 1 : 0;
    return cuda_status(launch_pdl(gather_rows_kernel, dim3((unsigned)n_idx), dim3(128), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<const unsigned char*>(table), idx, static_cast<unsigned char*>(out), row_bytes,
                                  n_table, vec16));
}

extern "C" int pimb200_scatter_rows(void* table, const long long* idx, const void* src, long n_idx, size_t row_bytes,
                                    long n_table, void* stream) {
    if (n_idx == 0 || row_bytes == 0) return PIMB200_OK;
    if (!table || !idx || !src || n_idx < 0 || n_idx > 0x7fffffffL || n_table <= 0) return PIMB200_ERR_BAD_ARG;
    const int vec16 = (row_bytes % 16 == 0 && aligned16(table) && aligned16(src)) ? 1 : 0;
    return cuda_status(launch_pdl(scatter_rows_kernel, dim3((unsigned)n_idx), dim3(128), 0, static_cast<cudaStream_t>(stream),
                                  static_cast<unsigned char*>(table), idx, static_cast<const unsigned char*>(src), row_bytes,
                                  n_table, vec16));
}

extern "C" int pimb200_attention_row(const void* q, const void* K, const void* V, const long long* len_dev, long len_add,
                                     long max_len, void* out, int heads, int head_dim, long kv_stride, float scale,
                                     void* stream) {
    if (!q || !K || !V || !out || heads <= 0 || head_dim <= 0 || max_len <= 0 || kv_stride < (long)heads * head_dim)
        return PIMB200_ERR_BAD_ARG;
    if (max_len > kAttnMaxLen || head_dim > 1024) return PIMB200_ERR_UNSUPPORTED;
    const size_t smem = ((size_t)max_len + (size_t)(kAttnThreads / 32) * head_dim) * sizeof(float);
    // the kernel runs within the default 48 KB of shared memory per CTA (16 B of it static): larger score / partial
    // buffers are refused here instead of failing at launch
    if (smem + 16 > 48 * 1024) return PIMB200_ERR_UNSUPPORTED;
    attention_row_kernel<<<(unsigned)heads, kAttnThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(q), static_cast<const __half*>(K), static_cast<const __half*>(V), len_dev, len_add,
        max_len, static_cast<__half*>(out), head_dim, kv_stride, scale);
    return launch_status();
}

extern "C" int pimb200_attention_rows(const void* q, const void* K, const void* V, const long long* len_dev, long len_inc,
                                      long len_add, long max_len, void* out, int n_seq, int heads, int head_dim,
                                      long kv_stride, long seq_stride, long q_stride, long out_stride, float scale,
                                      void* stream) {
    return pimb200_attention_rows_packed(q, K, V, nullptr, len_dev, len_inc, len_add, max_len, out, n_seq, heads, head_dim, kv_stride,
                                         seq_stride, q_stride, out_stride, scale, stream);
}

extern "C" int pimb200_attention_rows_packed(const void* q, const void* K, const void* V, const long long* row0, const long long* len_dev,
                                             long len_inc, long len_add, long max_len, void* out, int n_seq, int heads,
                                             int head_dim, long kv_stride, long seq_stride, long q_stride, long out_stride,
                                             float scale, void* stream) {
    if (n_seq == 0) return PIMB200_OK;
    if (!q || !K || !V || !out || n_seq < 0 || n_seq > 65535 || heads <= 0 || head_dim <= 0 || max_len <= 0 ||
        kv_stride < (long)heads * head_dim || seq_stride < 0 || len_inc < 0 || q_stride < (long)heads * head_dim ||
        out_stride < (long)heads * head_dim)
        return PIMB200_ERR_BAD_ARG;
    if (max_len > kAttnMaxLen || head_dim > 1024) return PIMB200_ERR_UNSUPPORTED;
    const int rc = launch_attention_decode(static_cast<const __half*>(q), static_cast<const __half*>(K), static_cast<const __half*>(V),
                                           row0, len_dev, len_inc, len_add, max_len, static_cast<__half*>(out), n_seq, heads,
                                           head_dim, kv_stride, seq_stride, q_stride, out_stride, scale, static_cast<cudaStream_t>(stream));
    if (rc != PIMB200_ERR_UNSUPPORTED) return rc;
    const size_t smem = ((size_t)max_len + (size_t)(kAttnThreads / 32) * head_dim) * sizeof(float);
    if (smem + 16 > 48 * 1024) return PIMB200_ERR_UNSUPPORTED;
    attention_rows_kernel<<<dim3((unsigned)heads, (unsigned)n_seq), kAttnThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(q), static_cast<const __half*>(K), static_cast<const __half*>(V), row0, len_dev, len_inc, len_add,
        max_len, static_cast<__half*>(out), head_dim, kv_stride, seq_stride, q_stride, out_stride, scale);
    return launch_status();
}

namespace {
template <int C, int PER_SM>
int launch_bahdanau(const __half* q, const __half* kp, const __half* values, const long long* lengths, const __half* v, const __half* bias,
                    __half* ctx, float* scores, int n_seq, long max_len, int H, long row_stride, long seq_stride, long ctx_stride, int copies,
                    long copy_stride, cudaStream_t st) {
    const size_t smem = ((size_t)2 * H + 8 * kBahdanauThreads + max_len) * sizeof(float);
    return cuda_status(launch_pdl<C>(bahdanau_kernel<C, PER_SM>, dim3(C, n_seq), dim3(kBahdanauThreads), smem, st, q, kp, values, lengths, v, bias, ctx,
                                     scores, max_len, H, row_stride, seq_stride, ctx_stride, copies, copy_stride));
}
}  // namespace

extern "C" int pimb200_additive_attention(const void* q, const void* keys_proj, const void* values, const long long* lengths,
                                          const void* v, const void* bias, void* ctx, float* scores, int n_seq,
                                          long max_len, int H, long row_stride, long seq_stride, long ctx_stride,
                                          void* stream) {
    return pimb200_additive_attention_copies(q, keys_proj, values, lengths, v, bias, ctx, scores, n_seq, max_len, H, row_stride, seq_stride,
                                             ctx_stride, 1, 0, stream);
}

extern "C" int pimb200_additive_attention_copies(const void* q, const void* keys_proj, const void* values, const long long* lengths,
                                                 const void* v, const void* bias, void* ctx, float* scores, int n_seq, long max_len,
                                                 int H, long row_stride, long seq_stride, long ctx_stride, int copies, long copy_stride,
                                                 void* stream) {
    if (n_seq == 0) return PIMB200_OK;
    if (copies < 1 || (copies > 1 && copy_stride < H)) return PIMB200_ERR_BAD_ARG;
    if (!q || !keys_proj || !values || !v || !ctx || !scores || n_seq < 0 || n_seq > 65535 || max_len <= 0 || H <= 0 ||
        row_stride < H || seq_stride < 0 || ctx_stride < H)
        return PIMB200_ERR_BAD_ARG;
    if ((size_t)max_len * sizeof(float) + 64 > 48 * 1024) return PIMB200_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (H % 8 == 0 && row_stride % 8 == 0 && seq_stride % 8 == 0 && ctx_stride % 8 == 0 && copy_stride % 8 == 0 && aligned16(keys_proj) &&
        aligned16(values) && aligned16(ctx) && ((size_t)2 * H + 8 * kBahdanauThreads + max_len) * sizeof(float) + 64 <= 48 * 1024) {
        // CTAs per sentence: as many as are resident at once, if the pieces of a row split evenly: a CTA's own chain is what takes the
        // time.  Four per SM leave 64 registers a thread, which spills, so grids that three per SM hold have 80 (20 / 50 keys, us with
        // three / four per SM: 64 sentences 6.4 / 7.4 and 8.9 / 10.7; 104: 6.8 / 7.8 and 9.3 / 11.3; 200: 8.3 / 10.1 and 14.0 / 18.0;
        // 400: 11.4 / 14.3 and 23.0 / 29.6).  Clusters do not fill every SM: of four CTAs, 104 fit with three per SM (106: 10.8) and 141
        // with four (144: 11.4), of two CTAs all of 222 and 296.  More CTAs than are resident cost more than fewer CTAs per sentence
        // (128 sentences of 20 keys: 8.0 with four, 8.1 with two, 9.7 with one; 148: 12.7, 8.2, 7.0; 256: 10.4 with two, 11.0 with one)
        auto run = [&](auto f) {
            return f(static_cast<const __half*>(q), static_cast<const __half*>(keys_proj), static_cast<const __half*>(values), lengths,
                     static_cast<const __half*>(v), static_cast<const __half*>(bias), static_cast<__half*>(ctx), scores, n_seq, max_len, H,
                     row_stride, seq_stride, ctx_stride, copies, copy_stride, st);
        };
        auto fits = [&](int c) { return (H / 8) % c == 0 && H / 8 / c <= kBahdanauThreads && kBahdanauThreads % (H / 8 / c) == 0; };
        const long sms = kNumSmB200, n = n_seq, lost = 28;         // (CTAs that clusters of four leave out)
        if (fits(8) && 8 * n <= 2 * sms) return run(launch_bahdanau<8, 3>);
        if (fits(4) && 4 * n <= 4 * sms - lost) return 4 * n <= 3 * sms - lost ? run(launch_bahdanau<4, 3>) : run(launch_bahdanau<4, 4>);
        if (fits(2) && 2 * n <= 4 * sms) return 2 * n <= 3 * sms ? run(launch_bahdanau<2, 3>) : run(launch_bahdanau<2, 4>);
        if (fits(1)) return n <= 3 * sms ? run(launch_bahdanau<1, 3>) : run(launch_bahdanau<1, 4>);
    }
    const long rows = (long)n_seq * max_len;
    const int rc = cuda_status(launch_pdl(
        additive_scores_kernel, dim3((unsigned)((rows + kAddAttnThreads / 32 - 1) / (kAddAttnThreads / 32))), dim3(kAddAttnThreads), 0, st,
        static_cast<const __half*>(q), static_cast<const __half*>(keys_proj), lengths, static_cast<const __half*>(v),
        static_cast<const __half*>(bias), scores, n_seq, max_len, H, row_stride, seq_stride));
    if (rc != PIMB200_OK) return rc;
    return cuda_status(launch_pdl(
        additive_context_kernel, dim3((unsigned)((H + kAddAttnSlice - 1) / kAddAttnSlice), (unsigned)n_seq), dim3(kAddAttnSlice / 2),
        (size_t)max_len * sizeof(float), st, scores, static_cast<const __half*>(values), lengths, static_cast<__half*>(ctx), max_len, H,
        row_stride, seq_stride, ctx_stride, copies, copy_stride));
}

extern "C" int pimb200_add_layer_norm_rows(const void* x, const void* r, const void* gamma, const void* beta, void* y,
                                           long rows, long cols, float eps, void* stream) {
    if (rows == 0 || cols == 0) return PIMB200_OK;
    if (!x || !r || !y || !rows_ok(rows, cols)) return PIMB200_ERR_BAD_ARG;
    if (cols % 8 == 0 && cols <= 2048 && aligned16(x) && aligned16(r) && aligned16(y)) {
        const int warps = rows <= 4 * kNumSmB200 ? 1 : 8;
        const dim3 grid((unsigned)((rows + warps - 1) / warps)), block(warps * 32);
        auto run = [&](auto kernel) {
            return cuda_status(launch_pdl(kernel, grid, block, 0, static_cast<cudaStream_t>(stream), static_cast<const __half*>(x),
                                          static_cast<const __half*>(r), static_cast<const __half*>(gamma),
                                          static_cast<const __half*>(beta), static_cast<__half*>(y), rows, (int)cols, eps));
        };
        return cols <= 256 ? run(add_layer_norm_warp_kernel<1>) : cols <= 512 ? run(add_layer_norm_warp_kernel<2>)
             : cols <= 1024 ? run(add_layer_norm_warp_kernel<4>) : run(add_layer_norm_warp_kernel<8>);
    }
    if ((size_t)cols * sizeof(float) + 64 > 48 * 1024) return PIMB200_ERR_UNSUPPORTED;
    add_layer_norm_rows_kernel<128><<<(unsigned)rows, 128, (size_t)cols * sizeof(float), static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(x), static_cast<const __half*>(r), static_cast<const __half*>(gamma),
        static_cast<const __half*>(beta), static_cast<__half*>(y), cols, eps);
    return launch_status();
}

extern "C" int pimb200_attention_block(const void* q, const void* k, const void* v, const long long* lengths, void* out,
                                       int n_seq, long max_len, int heads, int head_dim, long row_stride, long seq_stride,
                                       long out_row_stride, long out_seq_stride, float scale, void* stream) {
    return pimb200_attention_block_packed(q, k, v, lengths, nullptr, out, n_seq, max_len, heads, head_dim, row_stride, seq_stride,
                                          out_row_stride, out_seq_stride, scale, stream);
}

extern "C" int pimb200_attention_block_packed(const void* q, const void* k, const void* v, const long long* lengths, const long long* row0,
                                              void* out, int n_seq, long max_len, int heads, int head_dim, long row_stride,
                                              long seq_stride, long out_row_stride, long out_seq_stride, float scale, void* stream) {
    if (n_seq == 0) return PIMB200_OK;
    if (!q || !k || !v || !out || n_seq < 0 || n_seq > 65535 || heads <= 0 || head_dim <= 0 || max_len <= 0 ||
        row_stride < (long)heads * head_dim || out_row_stride < (long)heads * head_dim || seq_stride < 0 || out_seq_stride < 0)
        return PIMB200_ERR_BAD_ARG;
    const int rc = launch_attention_block(static_cast<const __half*>(q), static_cast<const __half*>(k), static_cast<const __half*>(v),
                                          lengths, row0, static_cast<__half*>(out), n_seq, max_len, heads, head_dim, row_stride,
                                          seq_stride, out_row_stride, out_seq_stride, scale, static_cast<cudaStream_t>(stream));
    if (rc != PIMB200_ERR_UNSUPPORTED) return rc;
    const size_t smem = (size_t)max_len * (head_dim + 2) * 2 + (size_t)max_len * head_dim * 2 +
                        (size_t)(kBlockAttnThreads / 32) * (head_dim + max_len) * sizeof(float);
    if (smem > 48 * 1024 || head_dim % 2 != 0) return PIMB200_ERR_UNSUPPORTED;
    attention_block_kernel<<<dim3((unsigned)heads, (unsigned)n_seq), kBlockAttnThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(q), static_cast<const __half*>(k), static_cast<const __half*>(v), lengths, row0,
        static_cast<__half*>(out), max_len, head_dim, row_stride, seq_stride, out_row_stride, out_seq_stride, scale);
    return launch_status();
}

extern "C" int pimb200_topk_rows(const void* x, void* values, long long* idx, long rows, long cols, int k, int largest,
                                 void* stream) {
    if (rows == 0 || k == 0) return PIMB200_OK;
    if (!x || !values || !idx || !rows_ok(rows, cols) || k < 0) return PIMB200_ERR_BAD_ARG;
    if (k > cols) return PIMB200_ERR_BAD_ARG;
    if (k > 64) return PIMB200_ERR_UNSUPPORTED;      // k passes over the row: meant for beam widths, not for sorting
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cols >= kWideRow)
        topk_rows_kernel<1024><<<(unsigned)rows, 1024, 0, st>>>(static_cast<const __half*>(x), static_cast<__half*>(values), idx,
                                                               cols, k, largest ? 1 : 0);
    else
        topk_rows_kernel<128><<<(unsigned)rows, 128, 0, st>>>(static_cast<const __half*>(x), static_cast<__half*>(values), idx,
                                                             cols, k, largest ? 1 : 0);
    return launch_status();
}
