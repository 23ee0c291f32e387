// The end of a greedy decode step for streams in lock step: vocabulary projection, arg max and the next step's embedding in
// two launches.  The projection's epilogue keeps only the largest logit of each row and tile, so the logits (131 MB per
// step at 2048 x 32000) are neither written nor read again, and the second launch reduces those pieces, stores the token
// and fetches its embedding row (plus a position row), which were three launches.
#include "common.cuh"
#include "gemm_rows.cuh"

namespace pimb200 {

int launch_skinny_argmax(const __half* W, const __half* X, const __half* bias, float* best_v, int* best_i, int* parts, int N, int K,
                         int J, int ldx, cudaStream_t st);

namespace {

constexpr int kRows = 8;            // streams per CTA: their pieces are whole 32-byte sectors
constexpr int kMaxParts = 2 * kNumSmB200;   // of the few-row projection: its CTAs

// SLICES threads share a row's pieces: 32 for many rows, 128 for few (all their loads in flight at once)
template <int SLICES>
__global__ void __launch_bounds__(kRows * SLICES) greedy_token_kernel(const float* best_v, const int* best_i,
                                                                       int parts, int J, int N, long long* __restrict__ idx,
                                                                       const __half* emb, const __half* pos,
                                                                       __half* __restrict__ x_next, int d, const long long* step,
                                                                       long long* next_step) {
    constexpr int WARPS = kRows * SLICES / 32;
    __shared__ float sv[WARPS][kRows];
    __shared__ int si[WARPS][kRows];
    __shared__ int tok[kRows];
    pdl_launch_dependents();
    pdl_wait();
    const long long at_step = step ? *step : 0;
    const int r = threadIdx.x % kRows, slice = threadIdx.x / kRows, j = blockIdx.x * kRows + r;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float v = -INFINITY;
    int i = 0x7fffffff;
    if (j < J) {
#pragma unroll 4
        for (int p = slice; p < parts; p += SLICES) {
            const float pv = best_v[(size_t)p * J + j];
            const int pi = best_i[(size_t)p * J + j];
            if (pv > v || (pv == v && pi < i)) { v = pv; i = pi; }   // the lowest index among equal maxima
        }
    }
#pragma unroll
    for (int o = kRows; o < 32; o <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
    }
    if (lane < kRows) { sv[warp][lane] = v; si[warp][lane] = i; }
    __syncthreads();
    if (threadIdx.x < kRows) {
#pragma unroll
        for (int w = 0; w < WARPS; ++w)
            if (sv[w][r] > v || (sv[w][r] == v && si[w][r] < i)) { v = sv[w][r]; i = si[w][r]; }
        i = i < N ? i : 0;           // a row without a comparable logit: index 0, as arg max has it
        tok[r] = i;
        if (j < J) idx[(size_t)at_step * J + j] = i;
    }
    if (next_step && blockIdx.x == 0 && threadIdx.x == 0) *next_step = at_step + 1;   // (nobody reads it before this kernel has ended)
    if (!emb) return;
    __syncthreads();
    const int chunks = d >> 3;
    for (int c = threadIdx.x; c < kRows * chunks; c += kRows * SLICES) {
        const int row = c / chunks, at = c % chunks, jj = blockIdx.x * kRows + row;
        if (jj >= J) break;
        uint4 e = reinterpret_cast<const uint4*>(emb + (size_t)tok[row] * d)[at];
        if (pos) {
            const uint4 p = reinterpret_cast<const uint4*>(pos)[at];
            __half2* a = reinterpret_cast<__half2*>(&e);
            const __half2* b = reinterpret_cast<const __half2*>(&p);
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = __hadd2(a[k], b[k]);
        }
        reinterpret_cast<uint4*>(x_next + (size_t)jj * d)[at] = e;
    }
}

}  // namespace
}  // namespace pimb200

using namespace pimb200;

extern "C" size_t pimb200_greedy_token_workspace(int N, int J) {
    if (N <= 0 || J <= 0) return 0;
    const size_t parts = J <= 32 ? kMaxParts : gemm_rows_max_parts(N);
    return parts * J * (sizeof(float) + sizeof(int));
}

extern "C" int pimb200_greedy_token(const void* W, const void* X, const void* bias, int N, int K, int J, int ldx, void* workspace,
                                    long long* idx, const void* emb, const void* pos, void* x_next, int d, void* stream) {
    return pimb200_greedy_token_step(W, X, bias, N, K, J, ldx, workspace, idx, nullptr, nullptr, emb, pos, x_next, d, stream);
}

extern "C" int pimb200_greedy_token_step(const void* W, const void* X, const void* bias, int N, int K, int J, int ldx, void* workspace,
                                         long long* idx, const long long* step, long long* next_step, const void* emb,
                                         const void* pos, void* x_next, int d, void* stream) {
    if ((step != nullptr) != (next_step != nullptr) || (step && step == next_step)) return PIMB200_ERR_BAD_ARG;
    if (!W || !X || !workspace || !idx || N <= 0 || K <= 0 || J <= 0 || ldx < K || (emb && (!x_next || d <= 0))) return PIMB200_ERR_BAD_ARG;
    if (emb && (d % 8 != 0 || !aligned16(emb) || !aligned16(x_next) || (pos && !aligned16(pos)))) return PIMB200_ERR_UNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __half *w = static_cast<const __half*>(W), *x = static_cast<const __half*>(X), *b = static_cast<const __half*>(bias);
    float* best_v = static_cast<float*>(workspace);
    int parts = J <= 32 ? kMaxParts : gemm_rows_max_parts(N);
    int* best_i = reinterpret_cast<int*>(best_v + (size_t)parts * J);
    const int rc = J <= 32 ? launch_skinny_argmax(w, x, b, best_v, best_i, &parts, N, K, J, ldx, st)
                           : launch_gemm_rows_argmax(w, x, b, best_v, best_i, &parts, N, K, J, ldx, st);
    if (rc != PIMB200_OK) return rc;
    auto run = [&](auto kernel, int slices) {
        return cuda_status(launch_pdl(kernel, dim3(ceil_div(J, kRows)), dim3(kRows * slices), 0, st, best_v, best_i, parts, J, N, idx,
                                      static_cast<const __half*>(emb), static_cast<const __half*>(pos), static_cast<__half*>(x_next), d, step,
                                      next_step));
    };
    return J <= 256 ? run(greedy_token_kernel<128>, 128) : run(greedy_token_kernel<32>, 32);
}
