// Attention kernels of the Transformer path for head widths of 64 and 128 (fp16 storage, fp32 softmax and sums):
// the single-query form of a decode step and the block form of an encoder layer.  Other head widths and unaligned rows
// take the kernels of rowops.cu.
#include "attention.cuh"

#include <math_constants.h>

#include "common.cuh"

namespace pimb200 {
namespace {

// ---------------------------------------------------------------------------------------------
// Decode step: one query per (head, sequence), a warp each, keys and values streamed once.
//
// HD / 8 lanes hold one key row (16 bytes each), so a load instruction of the warp covers four rows (two for HD = 128) of
// whole 128-byte lines; a lane per row reads 16 bytes of each of 32 lines and relies on L1 to keep them for the next
// seven loads, which it cannot with 64 warps of 8 KB each (3.0 TB/s at 2048 sequences, 5.1 now).  Rows go in chunks of CL
// loads of keys and of values in flight together; the softmax is the running one (maximum and sum rescaled from chunk to
// chunk).  The lanes of a row share its score after a shuffle reduction and hold the same columns of V, so weights need no
// exchange either; the row groups' partial outputs meet in the end.
// ---------------------------------------------------------------------------------------------
struct DecodeState {
    float m, sum, acc[8];
};

// rows c0 .. c0 + CL * 32 / (HD / 8) - 1 of one head; rows past L repeat the last one's key and are without weight
template <int HD, int CL>
__device__ __forceinline__ void decode_chunk(DecodeState& st, const float* qf, const __half* Ks, const __half* Vs, long c0, long L,
                                             long kv_stride, int grp) {
    constexpr int LPR = HD / 8, RPL = 32 / LPR;
    uint4 kr[CL], vr[CL];
#pragma unroll
    for (int i = 0; i < CL; ++i) {
        const long t = c0 + i * RPL + grp, at = (t < L ? t : L - 1) * kv_stride;
        kr[i] = ld_stream_v4(Ks + at);
        vr[i] = ld_stream_v4(Vs + at);
    }
    float s[CL], cm = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < CL; ++i) {
        s[i] = dot8f(kr[i], qf, 0.f);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
        if (c0 + i * RPL + grp >= L) s[i] = -CUDART_INF_F;
        cm = fmaxf(cm, s[i]);
    }
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
    // exp(-inf) = 0 in the first chunk.  While every score so far is -inf there is nothing to rescale, and -inf - -inf would be
    // a NaN that later scores cannot replace; the reference is 0 then, so that the weights are 0 as well
    const float mn = fmaxf(st.m, cm), ref = mn == -CUDART_INF_F ? 0.f : mn, keep = expf(st.m - ref);
    st.m = mn;
    st.sum *= keep;
#pragma unroll
    for (int e = 0; e < 8; ++e) st.acc[e] *= keep;
#pragma unroll
    for (int i = 0; i < CL; ++i) {
        const float p = expf(s[i] - ref);
        st.sum += p;
        if (c0 + i * RPL + grp >= L) vr[i] = make_uint4(0u, 0u, 0u, 0u);   // (0 x inf is a NaN)
        float vf[8];
        widen8(vr[i], vf);
#pragma unroll
        for (int e = 0; e < 8; ++e) st.acc[e] = fmaf(p, vf[e], st.acc[e]);
    }
}

template <int HD, int CL>
__global__ void __launch_bounds__(128) attention_decode_kernel(const __half* q, const __half* K,
                                                               const __half* V, const long long* row0, const long long* len_dev,
                                                               long len_inc, long len_add, long max_len, __half* __restrict__ out,
                                                               int heads, int n_seq, long kv_stride, long seq_stride, long q_stride,
                                                               long out_stride, float scale) {
    constexpr int LPR = HD / 8;              // lanes per row
    constexpr int RPL = 32 / LPR;            // rows per load instruction
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, sub = lane % LPR, grp = lane / LPR;
    const long task = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   // head fastest: a sequence's heads share lines
    if (task >= (long)heads * n_seq) return;
    const int h = (int)(task % heads), seq = (int)(task / heads);
    long L = (len_dev ? (long)len_dev[(size_t)seq * len_inc] : 0) + len_add;
    L = L < 0 ? 0 : (L > max_len ? max_len : L);
    const size_t at0 = (row0 ? (size_t)row0[seq] * kv_stride : (size_t)seq * seq_stride) + (size_t)h * HD + sub * 8;
    const __half *Ks = K + at0, *Vs = V + at0;
    float qf[8];
    DecodeState ds;
    ds.m = -CUDART_INF_F;
    ds.sum = 0.f;
    widen8(*reinterpret_cast<const uint4*>(q + (size_t)seq * q_stride + (size_t)h * HD + sub * 8), qf);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        qf[e] *= scale;
        ds.acc[e] = 0.f;
    }
    for (long c0 = 0; c0 < L;) {      // the chunk of 8, 4 or 2 loads that the rows left nearly fill
        const long left = L - c0;
        if (CL > 4 && left > 6 * RPL) { decode_chunk<HD, 8>(ds, qf, Ks, Vs, c0, L, kv_stride, grp); c0 += 8 * RPL; }
        else if (CL > 2 && left > 2 * RPL) { decode_chunk<HD, 4>(ds, qf, Ks, Vs, c0, L, kv_stride, grp); c0 += 4 * RPL; }
        else { decode_chunk<HD, 2>(ds, qf, Ks, Vs, c0, L, kv_stride, grp); c0 += 2 * RPL; }
    }
    float sum = ds.sum, *acc = ds.acc;
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    }
    if (grp == 0) {
        const float inv = L > 0 ? 1.0f / sum : 0.f;
        __half2 o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = __floats2half2_rn(acc[2 * e] * inv, acc[2 * e + 1] * inv);
        *reinterpret_cast<uint4*>(out + (size_t)seq * out_stride + (size_t)h * HD + sub * 8) = *reinterpret_cast<uint4*>(o);
    }
}

}  // namespace

namespace {

// ---------------------------------------------------------------------------------------------
// Encoder layer: every position of a padded sequence attends to its live positions, a CTA per (head, sequence).
//
// Up to 128 positions: queries, keys and values of the head sit in shared memory (rows padded by 16 bytes: conflict-free
// ldmatrix), and a warp takes 16 query rows at a time through two tensor-core products, S = Q K^T and O = P V, with the
// whole row of scores in registers between them.  A weight is kept as the sum of two fp16 numbers, so O has the precision
// of fp32 weights.  (An infinite value meets the first of them alone: the second may be zero or below.)  The work is 4 * L * L * HD flops per 8 * L * HD bytes, so HBM bounds it; with scalar products from
// shared memory the 2048 x 8 heads of 64 positions took 1116 us per layer (550 MB).
// ---------------------------------------------------------------------------------------------
constexpr int kBlockWarps = 4;

__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two weights as fp16 pairs: hi rounded, lo what the rounding left
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// The same for a product with infinite values: no weight above zero has a hi of zero (0 x inf is a NaN)
__device__ __forceinline__ void split2_nonzero(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    if (a > 0.f && (hi & 0xffffu) == 0u) hi |= 1u;
    if (b > 0.f && (hi >> 16) == 0u) hi |= 0x10000u;
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ bool has_infinity(uint32_t w) { return (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u; }   // or a NaN
__device__ __forceinline__ uint32_t finite_or_zero(uint32_t w) {
    if ((w & 0x7c00u) == 0x7c00u) w &= 0xffff0000u;
    if ((w & 0x7c000000u) == 0x7c000000u) w &= 0xffffu;
    return w;
}

template <int HD, int KT>   // KT: tiles of 16 positions
__global__ void __launch_bounds__(kBlockWarps * 32) attention_block_mma_kernel(
    const __half* Q, const __half* K, const __half* V, const long long* lengths,
    const long long* row0, __half* __restrict__ out, long max_len, long row_stride, long seq_stride, long out_row_stride,
    long out_seq_stride, float scale) {
    constexpr int PITCH = HD * 2 + 16;                  // bytes per shared row
    constexpr int CPR = HD / 8;                         // 16-byte chunks per row
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.x, seq = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long Ll = lengths ? (long)lengths[seq] : max_len;
    const int L = (int)(Ll < 0 ? 0 : (Ll > max_len ? max_len : Ll));
    const int tiles = (L + 15) >> 4, rows = tiles * 16;
    const size_t base = (row0 ? (size_t)row0[seq] * row_stride : (size_t)seq * seq_stride) + (size_t)h * HD;
    unsigned char *sQ = smem, *sK = smem + (size_t)KT * 16 * PITCH, *sV = sK + (size_t)KT * 16 * PITCH;
    bool infinite = false;      // a value is an infinity or a NaN: it meets the hi terms alone
    for (int i = threadIdx.x; i < rows * CPR; i += kBlockWarps * 32) {
        const int r = i / CPR, c = i % CPR;
        const size_t at = base + (size_t)r * row_stride + c * 8;
        uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a, d = a;
        if (r < L) {
            a = ld_stream_v4(Q + at);
            b = ld_stream_v4(K + at);
            d = ld_stream_v4(V + at);
            infinite = infinite || has_infinity(d.x) || has_infinity(d.y) || has_infinity(d.z) || has_infinity(d.w);
        }
        *reinterpret_cast<uint4*>(sQ + r * PITCH + c * 16) = a;
        *reinterpret_cast<uint4*>(sK + r * PITCH + c * 16) = b;
        *reinterpret_cast<uint4*>(sV + r * PITCH + c * 16) = d;
    }
    infinite = __syncthreads_or(infinite);
    __half* o = out + (row0 ? (size_t)row0[seq] * out_row_stride : (size_t)seq * out_seq_stride) + (size_t)h * HD;
    const uint32_t q0 = (uint32_t)__cvta_generic_to_shared(sQ), k0 = (uint32_t)__cvta_generic_to_shared(sK), v0 = (uint32_t)__cvta_generic_to_shared(sV);
    // ldmatrix rows of a lane: A and V take rows lane % 16 at column half lane / 16; K takes eight keys per matrix
    const uint32_t arow = (uint32_t)((lane & 15) * PITCH + (lane >> 4) * 16);
    const uint32_t krow = (uint32_t)(((lane & 7) + ((lane >> 4) << 3)) * PITCH + ((lane >> 3) & 1) * 16);
    for (int qt = warp; qt < tiles; qt += kBlockWarps) {
        uint32_t qa[HD / 16][4];
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) ldsm4(qa[k], q0 + qt * 16 * PITCH + arow + k * 32);
        float s[KT][2][4];
        float mx0 = -CUDART_INF_F, mx1 = -CUDART_INF_F;
#pragma unroll
        for (int t = 0; t < KT; ++t) {
            if (t < tiles) {
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[t][n][e] = 0.f;
#pragma unroll
                for (int k = 0; k < HD / 16; ++k) {
                    uint32_t kb[4];
                    ldsm4(kb, k0 + t * 16 * PITCH + krow + k * 32);
                    mma_16816(s[t][0], qa[k], kb[0], kb[1]);
                    mma_16816(s[t][1], qa[k], kb[2], kb[3]);
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int key = t * 16 + n * 8 + (lane & 3) * 2 + (e & 1);
                        s[t][n][e] = key < L ? s[t][n][e] * scale : -CUDART_INF_F;
                    }
                mx0 = fmaxf(mx0, fmaxf(fmaxf(s[t][0][0], s[t][0][1]), fmaxf(s[t][1][0], s[t][1][1])));
                mx1 = fmaxf(mx1, fmaxf(fmaxf(s[t][0][2], s[t][0][3]), fmaxf(s[t][1][2], s[t][1][3])));
            }
        }
#pragma unroll
        for (int x = 1; x <= 2; x <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, x));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, x));
        }
        float sum0 = 0.f, sum1 = 0.f, acc[HD / 8][4];
#pragma unroll
        for (int n = 0; n < HD / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
#pragma unroll
        for (int t = 0; t < KT; ++t) {
            if (t < tiles) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    s[t][n][0] = expf(s[t][n][0] - mx0); s[t][n][1] = expf(s[t][n][1] - mx0);
                    s[t][n][2] = expf(s[t][n][2] - mx1); s[t][n][3] = expf(s[t][n][3] - mx1);
                    sum0 += s[t][n][0] + s[t][n][1];
                    sum1 += s[t][n][2] + s[t][n][3];
                }
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float a = s[t][i >> 1][2 * (i & 1)], b = s[t][i >> 1][2 * (i & 1) + 1];
                    if (infinite) split2_nonzero(a, b, hi[i], lo[i]);
                    else split2(a, b, hi[i], lo[i]);
                }
#pragma unroll
                for (int n = 0; n < HD / 16; ++n) {
                    uint32_t vb[4];
                    ldsm4_trans(vb, v0 + t * 16 * PITCH + arow + n * 32);
                    mma_16816(acc[2 * n], hi, vb[0], vb[1]);
                    mma_16816(acc[2 * n + 1], hi, vb[2], vb[3]);
                    if (infinite)
#pragma unroll
                        for (int i = 0; i < 4; ++i) vb[i] = finite_or_zero(vb[i]);
                    mma_16816(acc[2 * n], lo, vb[0], vb[1]);
                    mma_16816(acc[2 * n + 1], lo, vb[2], vb[3]);
                }
            }
        }
#pragma unroll
        for (int x = 1; x <= 2; x <<= 1) {
            sum0 += __shfl_xor_sync(0xffffffffu, sum0, x);
            sum1 += __shfl_xor_sync(0xffffffffu, sum1, x);
        }
        const float i0 = 1.0f / sum0, i1 = 1.0f / sum1;
        // the outputs go through the warp's own query rows, which it has read, to leave as whole 16-byte pieces
        __syncwarp();
        unsigned char* so = sQ + (size_t)qt * 16 * PITCH;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) {
            *reinterpret_cast<__half2*>(so + (lane >> 2) * PITCH + n * 16 + (lane & 3) * 4) = __floats2half2_rn(acc[n][0] * i0, acc[n][1] * i0);
            *reinterpret_cast<__half2*>(so + ((lane >> 2) + 8) * PITCH + n * 16 + (lane & 3) * 4) = __floats2half2_rn(acc[n][2] * i1, acc[n][3] * i1);
        }
        __syncwarp();
        for (int i = lane; i < 16 * CPR; i += 32) {
            const int r = i / CPR, c = i % CPR;
            if (qt * 16 + r < L)
                *reinterpret_cast<uint4*>(o + (size_t)(qt * 16 + r) * out_row_stride + c * 8) = *reinterpret_cast<const uint4*>(so + r * PITCH + c * 16);
        }
    }
    if (row0) return;                                                                         // packed rows: there are none past the length
    for (long i = (long)L * CPR + threadIdx.x; i < max_len * CPR; i += kBlockWarps * 32)      // rows past the length
        *reinterpret_cast<uint4*>(o + (size_t)(i / CPR) * out_row_stride + (i % CPR) * 8) = make_uint4(0u, 0u, 0u, 0u);
}

template <int HD, int KT>
int launch_block(const __half* q, const __half* k, const __half* v, const long long* lengths, const long long* row0, __half* out, int n_seq, long max_len,
                 int heads, long row_stride, long seq_stride, long out_row_stride, long out_seq_stride, float scale, cudaStream_t st) {
    constexpr size_t smem = (size_t)3 * KT * 16 * (HD * 2 + 16);
    static bool attr_set[64];                           // cudaFuncSetAttribute is per device
    if (smem > 48 * 1024) {
        int dev = 0;
        PIMB200_CUDA_TRY(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64) return PIMB200_ERR_UNSUPPORTED;
        if (!attr_set[dev]) {
            PIMB200_CUDA_TRY(cudaFuncSetAttribute(attention_block_mma_kernel<HD, KT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            attr_set[dev] = true;
        }
    }
    return cuda_status(launch_pdl(attention_block_mma_kernel<HD, KT>, dim3(heads, n_seq), dim3(kBlockWarps * 32), smem, st, q, k, v,
                                  lengths, row0, out, max_len, row_stride, seq_stride, out_row_stride, out_seq_stride, scale));
}

}  // namespace

int launch_attention_block(const __half* q, const __half* k, const __half* v, const long long* lengths, const long long* row0, __half* out, int n_seq,
                           long max_len, int heads, int head_dim, long row_stride, long seq_stride, long out_row_stride,
                           long out_seq_stride, float scale, cudaStream_t st) {
    if ((head_dim != 64 && head_dim != 128) || max_len > 128 || row_stride % 8 || seq_stride % 8 || out_row_stride % 8 ||
        out_seq_stride % 8 || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out))
        return PIMB200_ERR_UNSUPPORTED;
    auto run = [&](auto f) {
        return f(q, k, v, lengths, row0, out, n_seq, max_len, heads, row_stride, seq_stride, out_row_stride, out_seq_stride, scale, st);
    };
    if (head_dim == 64) return max_len <= 64 ? run(launch_block<64, 4>) : run(launch_block<64, 8>);
    return max_len <= 64 ? run(launch_block<128, 4>) : run(launch_block<128, 8>);
}

int launch_attention_decode(const __half* q, const __half* K, const __half* V, const long long* row0, const long long* len_dev, long len_inc,
                            long len_add, long max_len, __half* out, int n_seq, int heads, int head_dim, long kv_stride,
                            long seq_stride, long q_stride, long out_stride, float scale, cudaStream_t st) {
    if ((head_dim != 64 && head_dim != 128) || kv_stride % 8 || seq_stride % 8 || q_stride % 8 || out_stride % 8 || !aligned16(q) ||
        !aligned16(K) || !aligned16(V) || !aligned16(out))
        return PIMB200_ERR_UNSUPPORTED;
    const long tasks = (long)heads * n_seq;
    // few queries: one warp per CTA, so that they spread over the SMs; many: four
    const int warps = tasks <= 4 * kNumSmB200 ? 1 : 4;
    const dim3 grid((unsigned)((tasks + warps - 1) / warps)), block(warps * 32);
    auto run = [&](auto kernel) {
        return cuda_status(launch_pdl(kernel, grid, block, 0, st, q, K, V, row0, len_dev, len_inc, len_add, max_len, out, heads, n_seq, kv_stride,
                                      seq_stride, q_stride, out_stride, scale));
    };
    // the longest attended length that the host knows of decides how many rows a warp has in flight (and its registers)
    const long longest = len_dev ? max_len : len_add, rows = 256 / head_dim;      // rows per load
    if (head_dim == 64)
        return longest <= 2 * rows ? run(attention_decode_kernel<64, 2>) : longest <= 6 * rows ? run(attention_decode_kernel<64, 4>)
                                                                                     : run(attention_decode_kernel<64, 8>);
    return longest <= 6 * rows ? run(attention_decode_kernel<128, 4>) : run(attention_decode_kernel<128, 8>);
}

}  // namespace pimb200
