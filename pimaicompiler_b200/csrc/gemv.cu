// Batch-1 GEMV family, the SIMT GEMM fall-back and the fp16 glue ops.
//
// These kernels stand where the reference offloads to PIM-HBM (PimExecuteGemm) or launches its
// HIP GEMV templates (runtime/include/executor/op_executor/custom_ops.h).  All of them are
// HBM-bandwidth bound: 128-bit coalesced loads that bypass L1, fp32 accumulation, warp-shuffle
// reductions and the bias / ReLU epilogue fused into the same kernel.
#include <atomic>
#include <mutex>
#include <type_traits>

#include "batch_plan.h"
#include "common.cuh"

namespace pimb200 {

// =============================================================================================
// MV:  y[n] = act(sum_k W[n,k] x[k] + b[n])
// One warp owns R consecutive rows; a lane walks the row in 16-byte chunks (stride 32 chunks),
// so a warp reads 512 contiguous bytes per row per iteration.  W bypasses L1 (read once); x is
// read through L1 (it is a few KB and every warp reads all of it) — staging it in shared memory
// first costs a barrier before the first weight load and measured slower.  R*unroll independent
// 16-byte loads are in flight per lane.
// =============================================================================================
template <int R>
__device__ __forceinline__ void mv_finish(float (&acc)[R], const __half* bias, __half* y, int row0, int N, int act, int lane) {
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = warp_sum(acc[r]);
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            int row = row0 + r;
            if (row < N) {
                float v = acc[r] + (bias ? __half2float(bias[row]) : 0.f);
                if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
                y[row] = __float2half_rn(v);
            }
        }
    }
}

template <int R>
__global__ void __launch_bounds__(256) gemv_mv_vec_kernel(const __half* __restrict__ W, const __half* __restrict__ x,
                                                          const __half* __restrict__ bias, __half* __restrict__ y,
                                                          int N, int K, int act) {
    const int K8 = K >> 3;
    const uint4* x4 = reinterpret_cast<const uint4*>(x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = (blockIdx.x * (blockDim.x >> 5) + warp) * R;
    if (row0 >= N) return;

    const uint4* wrow[R];
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        int row = min(row0 + r, N - 1);  // clamp: rows past N re-read the last row, never stored
        wrow[r] = reinterpret_cast<const uint4*>(W + (size_t)row * K);
        acc[r] = 0.f;
    }
#pragma unroll 4
    for (int c = lane; c < K8; c += 32) {
        float xf[8];
        widen8(__ldg(x4 + c), xf);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = dot8f(ldg_stream_v4(wrow[r] + c), xf, acc[r]);
    }
    mv_finish<R>(acc, bias, y, row0, N, act, lane);
}

// The same for small matrices, where start and ramp are half the time.  The launch may start while its predecessor is still
// running: it then asks for its rows of W to be brought into L2 (which is coherent, so it does not matter whether anyone still
// writes them) and reads everything behind the wait, by plain loads.  The launcher leaves room on an SM for this launch's share of CTAs
// and one more: where registers allow six and the grid is two per SM, CTAs that start as their predecessors leave pile up on some
// SMs.  In a loop of launches, W in HBM / in L2, us, kernel above, this one with room for six, and as it is:
//   1024 x 1024 2.78 / 2.19, 2.27 / 1.90, 1.95 / 1.74    2000 x 4096 6.6 / 4.3, 6.5 / 5.8, 5.3 / 4.0
//   4096 x 1024 3.62 / 2.70, 3.09 / 2.66, 2.62 / 2.35    5000 x 1024 4.5 / 2.7, 4.0 / 3.4, 3.9 / 2.8
// (Room for exactly its share is faster still in such a loop and slower among other launches, which find no room beside it: a cell's
// step behind it 8.8 us in all, 10.1.)
// From 8 M elements on the read-only path of the former counts for more: 16384 x 1024 7.40, 7.66 here; 32320 x 1024 12.7, 13.5;
// 32768 x 4096 42.5, 45.9.
constexpr size_t kMvEarlyMax = (size_t)8 << 20;     // elements
constexpr int kMvMaxPerSm = 5;                      // (registers allow no more than six)
template <int R>
__global__ void __launch_bounds__(256) gemv_mv_early_kernel(const __half* W, const __half* x, const __half* bias, __half* y, int N, int K, int act) {
    pdl_launch_dependents();
    const int K8 = K >> 3;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = (blockIdx.x * (blockDim.x >> 5) + warp) * R;
    if (lane < R && row0 + lane < N) prefetch_l2(W + (size_t)(row0 + lane) * K, (uint32_t)K * 2);
    pdl_wait();
    if (row0 >= N) return;

    const uint4* wrow[R];
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        wrow[r] = reinterpret_cast<const uint4*>(W + (size_t)min(row0 + r, N - 1) * K);
        acc[r] = 0.f;
    }
#pragma unroll 4
    for (int c = lane; c < K8; c += 32) {
        float xf[8];
        widen8(ld_v4(x + 8 * c), xf);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = dot8f(ld_stream_v4(wrow[r] + c), xf, acc[r]);
    }
    mv_finish<R>(acc, bias, y, row0, N, act, lane);
}

// any K, any alignment: one warp per row, scalar half loads
__global__ void __launch_bounds__(256) gemv_mv_generic_kernel(const __half* __restrict__ W, const __half* __restrict__ x,
                                                              const __half* __restrict__ bias, __half* __restrict__ y,
                                                              int N, int K, int act) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= N) return;
    const __half* w = W + (size_t)row * K;
    float acc = 0.f;
    for (int k = lane; k < K; k += 32) acc = fmaf(__half2float(w[k]), __half2float(x[k]), acc);
    acc = warp_sum(acc);
    if (lane == 0) {
        float v = acc + (bias ? __half2float(bias[row]) : 0.f);
        if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        y[row] = __float2half_rn(v);
    }
}

static int launch_gemv_mv(const __half* W, const __half* x, const __half* bias, __half* y, int N, int K, int act,
                          cudaStream_t st) {
    const bool vec = (K % 8 == 0) && aligned16(W) && aligned16(x);
    if (!vec) {
        gemv_mv_generic_kernel<<<ceil_div(N, 8), 256, 0, st>>>(W, x, bias, y, N, K, act);
        return launch_status();
    }
    // rows per warp: enough warps to cover every SM several times, else fewer rows per warp
    const long warps4 = ((long)N + 3) / 4, warps2 = ((long)N + 1) / 2;
    const long want = (long)kNumSmB200 * 8 * 2;
    const int R = warps4 >= want ? 4 : (warps2 >= want ? 2 : 1);
    const int grid = ceil_div(N, 8 * R);
    if ((size_t)N * K < kMvEarlyMax) {
        static void (*const early[3])(const __half*, const __half*, const __half*, __half*, int, int, int) = {
            gemv_mv_early_kernel<1>, gemv_mv_early_kernel<2>, gemv_mv_early_kernel<4>};
        const auto fn = early[R / 2];
        // CTAs per SM, by an amount of shared memory that nothing uses: this launch's share and one more
        const int per_sm = ceil_div(grid, kNumSmB200) + 1;
        size_t room = 0;
        if (per_sm <= kMvMaxPerSm) {
            room = tc::kSmemPerSm / per_sm - 1024;             // (1 KB of a CTA's share is the system's)
            static std::atomic<bool> allowed[64][3];
            int dev = 0;
            PIMB200_CUDA_TRY(cudaGetDevice(&dev));
            if (dev >= 64 || !allowed[dev][R / 2].load(std::memory_order_relaxed)) {
                PIMB200_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(tc::kSmemPerSm / 2 - 1024)));
                if (dev < 64) allowed[dev][R / 2].store(true, std::memory_order_relaxed);
            }
        }
        return cuda_status(launch_pdl(fn, dim3(grid), dim3(256), room, st, W, x, bias, y, N, K, act));
    }
    if (R == 4) gemv_mv_vec_kernel<4><<<grid, 256, 0, st>>>(W, x, bias, y, N, K, act);
    else if (R == 2) gemv_mv_vec_kernel<2><<<grid, 256, 0, st>>>(W, x, bias, y, N, K, act);
    else gemv_mv_vec_kernel<1><<<grid, 256, 0, st>>>(W, x, bias, y, N, K, act);
    return launch_status();
}

// =============================================================================================
// VM:  y[n] = act(sum_k x[k] A[k,n] + b[n]),  A row-major [K,N]
// Threads run along n (8 columns = one 16-byte load each), so every row segment a warp touches
// is contiguous.  LPR lanes cover one row segment (LPR*8 columns); a warp covers 32/LPR rows
// per pass and the CTA's 8 warps cover 8*32/LPR rows.  K is additionally split over gridDim.y
// CTAs; their fp32 partial sums go through the per-device scratch and the CTA that draws the
// last ticket for a column tile reduces them and applies the epilogue.
// =============================================================================================
template <int LPR>
__global__ void __launch_bounds__(256) gemv_vm_vec_kernel(const __half* __restrict__ x, const __half* __restrict__ A,
                                                          const __half* __restrict__ bias, __half* __restrict__ y,
                                                          int K, int N, int act, int rows_per_split,
                                                          float* __restrict__ partials,
                                                          unsigned int* __restrict__ tickets) {
    constexpr int TILE = LPR * 8;        // columns per CTA
    constexpr int RPW = 32 / LPR;        // rows per warp per pass
    __shared__ float red[8][TILE];
    __shared__ int s_last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPR, cl = lane % LPR;
    const int col = blockIdx.x * TILE + cl * 8;
    const int S = gridDim.y, split = blockIdx.y;
    const int k0 = split * rows_per_split;
    const int k1 = min(K, k0 + rows_per_split);

    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    if (col < N) {
#pragma unroll 8
        for (int k = k0 + warp * RPW + sub; k < k1; k += 8 * RPW) {
            const uint4 a = ldg_stream_v4(A + (size_t)k * N + col);
            const float xk = __half2float(__ldg(x + k));
            float2 f;
            f = h2f2(a.x); acc[0] = fmaf(xk, f.x, acc[0]); acc[1] = fmaf(xk, f.y, acc[1]);
            f = h2f2(a.y); acc[2] = fmaf(xk, f.x, acc[2]); acc[3] = fmaf(xk, f.y, acc[3]);
            f = h2f2(a.z); acc[4] = fmaf(xk, f.x, acc[4]); acc[5] = fmaf(xk, f.y, acc[5]);
            f = h2f2(a.w); acc[6] = fmaf(xk, f.x, acc[6]); acc[7] = fmaf(xk, f.y, acc[7]);
        }
    }
    // fold the row groups of a warp together, then the warps through shared memory
#pragma unroll
    for (int o = 16; o >= LPR; o >>= 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    if (sub == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) red[warp][cl * 8 + j] = acc[j];
    }
    __syncthreads();
    const int t = threadIdx.x;
    const int ocol = blockIdx.x * TILE + t;
    float v = 0.f;
    if (t < TILE) {
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][t];
    }
    if (S > 1) {
        if (t < TILE && ocol < N) __stcg(partials + (size_t)split * N + ocol, v);
        __threadfence();
        __syncthreads();
        if (t == 0) {
            unsigned int tk = atomicAdd(tickets + blockIdx.x, 1u);
            s_last = (tk == (unsigned)(S - 1));
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        v = 0.f;
        if (t < TILE && ocol < N) {
            for (int s = 0; s < S; ++s) v += __ldcg(partials + (size_t)s * N + ocol);
        }
        if (t == 0) tickets[blockIdx.x] = 0;  // leave the ticket counter clean for the next call
    }
    if (t < TILE && ocol < N) {
        v += bias ? __half2float(bias[ocol]) : 0.f;
        if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        y[ocol] = __float2half_rn(v);
    }
}

// any N, any alignment: one thread per column, rows split across the 8 warps of a CTA
__global__ void __launch_bounds__(256) gemv_vm_generic_kernel(const __half* __restrict__ x, const __half* __restrict__ A,
                                                              const __half* __restrict__ bias, __half* __restrict__ y,
                                                              int K, int N, int act) {
    __shared__ float red[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = blockIdx.x * 32 + lane;
    float acc = 0.f;
    if (col < N)
        for (int k = warp; k < K; k += 8) acc = fmaf(__half2float(x[k]), __half2float(A[(size_t)k * N + col]), acc);
    red[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && col < N) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][lane];
        v += bias ? __half2float(bias[col]) : 0.f;
        if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        y[col] = __float2half_rn(v);
    }
}

// Chooses the column-tile width and the K split.  Exposed so the scratch-free entry point can
// reuse the same plan with its own scratch.
struct VmPlan {
    int lpr;             // lanes per row segment: 32 or 8
    int tiles;           // gridDim.x
    int splits;          // gridDim.y
    int rows_per_split;
};
VmPlan plan_gemv_vm(int K, int N, size_t max_partial_floats, int max_tiles) {
    VmPlan p;
    p.lpr = (ceil_div(N, 256) >= kNumSmB200 / 4) ? 32 : 8;
    const int tile = p.lpr * 8;
    p.tiles = ceil_div(N, tile);
    const int rows_per_pass = 8 * (32 / p.lpr);       // rows a CTA covers per pass
    int want = ceil_div(4 * kNumSmB200, p.tiles);     // about four CTAs per SM
    int max_by_rows = K / (rows_per_pass * 4);        // keep at least four passes per CTA
    if (max_by_rows < 1) max_by_rows = 1;
    int S = want < max_by_rows ? want : max_by_rows;
    if (S < 1) S = 1;
    if (p.tiles > max_tiles) S = 1;
    while (S > 1 && (size_t)S * (size_t)N > max_partial_floats) --S;
    p.rows_per_split = ceil_div(K, S);
    p.splits = ceil_div(K, p.rows_per_split);
    return p;
}

int launch_gemv_vm_with_scratch(const __half* x, const __half* A, const __half* bias, __half* y, int K, int N,
                                int act, const VmPlan& p, float* partials, unsigned int* tickets, cudaStream_t st) {
    dim3 grid(p.tiles, p.splits);
    if (p.lpr == 32)
        gemv_vm_vec_kernel<32><<<grid, 256, 0, st>>>(x, A, bias, y, K, N, act, p.rows_per_split, partials, tickets);
    else
        gemv_vm_vec_kernel<8><<<grid, 256, 0, st>>>(x, A, bias, y, K, N, act, p.rows_per_split, partials, tickets);
    return launch_status();
}

// The same for moderate K, in one phase: the S <= 8 CTAs that share a column tile are a cluster, whose partial sums
// meet in its first CTA's shared memory.  Through global memory (partial sums, a fence, a ticket, another trip to L2) the
// meeting took as long as the product itself, and the shared scratch needs an event behind every call.
template <int LPR, int S>
__global__ void __launch_bounds__(256) gemv_vm_cluster_kernel(const __half* x, const __half* A, const __half* bias, __half* y, int K, int N, int act,
                                                              int rows_per_split) {
    constexpr int TILE = LPR * 8, RPW = 32 / LPR, AHEAD = 8;
    __shared__ float red[8][TILE];
    __shared__ float parts[S][TILE];     // of the first CTA: every CTA's sums
    pdl_launch_dependents();
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPR, cl = lane % LPR;
    const int rank = blockIdx.x % S, tile = blockIdx.x / S;
    const int col = tile * TILE + cl * 8;
    const int k0 = rank * rows_per_split, k1 = min(K, k0 + rows_per_split);
    // the first rows on their way into L2 while the predecessor finishes (coherent: it does not matter who still writes them)
    if ((cl & 7) == 0 && col < N)
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int k = k0 + warp * RPW + sub + i * 8 * RPW;
            if (k < k1) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)k * N + col));
        }
    pdl_wait();
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    if (col < N) {
#pragma unroll 8
        for (int k = k0 + warp * RPW + sub; k < k1; k += 8 * RPW) {
            const uint4 a = ld_stream_v4(A + (size_t)k * N + col);
            const float xk = __half2float(x[k]);
            float2 f;
            f = h2f2(a.x); acc[0] = fmaf(xk, f.x, acc[0]); acc[1] = fmaf(xk, f.y, acc[1]);
            f = h2f2(a.y); acc[2] = fmaf(xk, f.x, acc[2]); acc[3] = fmaf(xk, f.y, acc[3]);
            f = h2f2(a.z); acc[4] = fmaf(xk, f.x, acc[4]); acc[5] = fmaf(xk, f.y, acc[5]);
            f = h2f2(a.w); acc[6] = fmaf(xk, f.x, acc[6]); acc[7] = fmaf(xk, f.y, acc[7]);
        }
    }
#pragma unroll
    for (int o = 16; o >= LPR; o >>= 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    if (sub == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) red[warp][cl * 8 + j] = acc[j];
    }
    __syncthreads();
    const int t = threadIdx.x, ocol = tile * TILE + t;
    float v = 0.f;
    if (t < TILE) {
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][t];
    }
    if (S > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");    // every CTA of the cluster has started
        if (t < TILE) {
            uint32_t at;
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(&parts[rank][t])));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank > 0) return;
        v = 0.f;
        if (t < TILE) {
#pragma unroll
            for (int s = 0; s < S; ++s) v += parts[s][t];
        }
    }
    if (t < TILE && ocol < N) {
        v += bias ? __half2float(bias[ocol]) : 0.f;
        if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        y[ocol] = __float2half_rn(v);
    }
}

// Column tile and slices of K: as many slices as keep every CTA resident at once (a second wave of a few CTAs costs as much as the
// first: 20000 columns x 4096 36.7 us with eight slices of 256 columns, 27.0 with seven, 29.3 by the split through memory), with at
// least four passes over the rows in each.  Narrow tiles hold 5.25 CTAs per SM (7000 x 4096: 770 CTAs 11.7..12.0 us, 660 12.6, 880
// 17.1), wide ones 4.  Wide tiles from where narrow ones would have less than four slices (12000 columns x 4096: 17.3 us in narrow
// ones, 18.9 in wide ones; 14000: 25.6 and 20.4), and up to K = 1024 from where they fill a quarter of the SMs (9480 x 512: 4.1 us,
// 5.1 in narrow ones).
struct VmSplit {
    bool wide;
    int tiles, slices;
};
static VmSplit split_vm(int K, int N) {
    const int narrow = ceil_div(N, 64);
    const int narrow_most = kNumSmB200 * 21 / 4;
    const bool wide = narrow * 4 > narrow_most || (K <= 1024 && ceil_div(N, 256) >= kNumSmB200 / 4);
    VmSplit v{wide, wide ? ceil_div(N, 256) : narrow, 8};
    const int passes = K / (wide ? 8 : 32), most = wide ? kNumSmB200 * 4 : narrow_most;
    while (v.slices > 1 && (v.tiles * v.slices > most || passes < 4 * v.slices)) --v.slices;
    return v;
}
template <int LPR>
static int launch_gemv_vm_cluster(const __half* x, const __half* A, const __half* bias, __half* y, int K, int N, int act, const VmSplit& v,
                                  cudaStream_t st) {
    const dim3 grid(v.tiles * v.slices), block(256);
    const int rows = ceil_div(K, v.slices);
    auto run = [&](auto slices) {
        constexpr int S = decltype(slices)::value;
        return cuda_status(launch_pdl<S>(gemv_vm_cluster_kernel<LPR, S>, grid, block, 0, st, x, A, bias, y, K, N, act, rows));
    };
    switch (v.slices) {
        case 1: return run(std::integral_constant<int, 1>());
        case 2: return run(std::integral_constant<int, 2>());
        case 3: return run(std::integral_constant<int, 3>());
        case 4: return run(std::integral_constant<int, 4>());
        case 5: return run(std::integral_constant<int, 5>());
        case 6: return run(std::integral_constant<int, 6>());
        case 7: return run(std::integral_constant<int, 7>());
        default: return run(std::integral_constant<int, 8>());
    }
}

static std::mutex g_vm_mutex;
static cudaStream_t g_vm_last_stream[64];
static bool g_vm_used[64];
static cudaEvent_t g_vm_event[64];   // recorded behind the last split-K user of the device's scratch

// Calls on one device share the split-K scratch.  Every split-K launch records an event behind itself on its own
// stream (scratch_user_done); a later caller on a different stream waits for that event first.  Nothing is ever
// recorded on a stream handle remembered from an earlier call (the caller may have destroyed it since).
// While a stream is being captured into a CUDA graph neither side is possible: captured launches are not ordered
// against other users of the scratch, so replays of graphs that contain split-K VM products must be ordered by
// the caller against every other VM call on the device.
static int order_scratch_users(int dev, cudaStream_t st) {
    if (dev < 0 || dev >= 64) return PIMB200_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lk(g_vm_mutex);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cs);
    if (cs != cudaStreamCaptureStatusNone) return PIMB200_OK;
    if (g_vm_used[dev] && g_vm_last_stream[dev] != st) PIMB200_CUDA_TRY(cudaStreamWaitEvent(st, g_vm_event[dev], 0));
    return PIMB200_OK;
}
static int scratch_user_done(int dev, cudaStream_t st) {
    if (dev < 0 || dev >= 64) return PIMB200_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lk(g_vm_mutex);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cs);
    if (cs != cudaStreamCaptureStatusNone) return PIMB200_OK;
    if (!g_vm_event[dev]) PIMB200_CUDA_TRY(cudaEventCreateWithFlags(&g_vm_event[dev], cudaEventDisableTiming));
    PIMB200_CUDA_TRY(cudaEventRecord(g_vm_event[dev], st));
    g_vm_used[dev] = true;
    g_vm_last_stream[dev] = st;
    return PIMB200_OK;
}

static int launch_gemv_vm(const __half* x, const __half* A, const __half* bias, __half* y, int K, int N, int act,
                          bool allow_split, cudaStream_t st) {
    const bool vec = (N % 8 == 0) && aligned16(A);
    if (!vec) {
        gemv_vm_generic_kernel<<<ceil_div(N, 32), 256, 0, st>>>(x, A, bias, y, K, N, act);
        return launch_status();
    }
    DeviceCtx* ctx = allow_split ? current_ctx() : nullptr;
    if (allow_split && !ctx) return PIMB200_ERR_NOT_INIT;
    // one phase up to K = 4096, and up to 8192 where its CTAs fill the SMs twice (1024 columns: 12.1 us, 10.5 with the split through
    // memory; 4096 columns: 15.2, 22.6)
    const VmSplit v = split_vm(K, N);
    if (K <= 4096 || (K <= 8192 && v.tiles * v.slices >= 2 * kNumSmB200))
        return v.wide ? launch_gemv_vm_cluster<32>(x, A, bias, y, K, N, act, v, st) : launch_gemv_vm_cluster<8>(x, A, bias, y, K, N, act, v, st);
    float* partials = nullptr;
    unsigned int* tickets = nullptr;
    VmPlan p;
    int dev = -1;
    if (allow_split) {
        p = plan_gemv_vm(K, N, kSplitKMaxFloats, kSplitKMaxTiles);
        if (p.splits > 1) {
            PIMB200_CUDA_TRY(cudaGetDevice(&dev));
            int rc = order_scratch_users(dev, st);
            if (rc != PIMB200_OK) return rc;
            partials = ctx->splitk_partials;
            tickets = ctx->splitk_tickets;
        }
    } else {
        p = plan_gemv_vm(K, N, 0, 0);  // forces a single split
    }
    const int rc = launch_gemv_vm_with_scratch(x, A, bias, y, K, N, act, p, partials, tickets, st);
    if (rc == PIMB200_OK && dev >= 0) return scratch_user_done(dev, st);
    return rc;
}

// =============================================================================================
// VV dot product: one CTA, fp32 accumulate
// =============================================================================================
__global__ void __launch_bounds__(256) dot_vv_kernel(const __half* __restrict__ a, const __half* __restrict__ b,
                                                     __half* __restrict__ y, int K) {
    __shared__ float red[8];
    float acc = 0.f;
    for (int k = threadIdx.x; k < K; k += blockDim.x) acc = fmaf(__half2float(a[k]), __half2float(b[k]), acc);
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w];
        y[0] = __float2half_rn(v);
    }
}

// =============================================================================================
// fp16 add, same-shape or row-broadcast, any n
// =============================================================================================
__global__ void __launch_bounds__(256) add_f16_vec_kernel(const uint4* A, const uint4* B,
                                                          uint4* C, size_t total8, int n8, int bcast) {
    pdl_launch_dependents();
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total8; i += (size_t)gridDim.x * blockDim.x) {
        uint4 a = A[i];
        uint4 b = B[bcast ? (i % n8) : i];
        uint4 c;
        __half2* ap = reinterpret_cast<__half2*>(&a);
        __half2* bp = reinterpret_cast<__half2*>(&b);
        __half2* cp = reinterpret_cast<__half2*>(&c);
#pragma unroll
        for (int j = 0; j < 4; ++j) cp[j] = __hadd2(ap[j], bp[j]);
        C[i] = c;
    }
}
__global__ void __launch_bounds__(256) add_f16_scalar_kernel(const __half* A, const __half* __restrict__ B,
                                                             __half* C, size_t total, int n, int bcast) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
        C[i] = __hadd(A[i], B[bcast ? (i % n) : i]);
}

// =============================================================================================
// strided copies (copy_ into a slice, cat along the inner dimension)
// =============================================================================================
template <typename V>
__global__ void __launch_bounds__(256) copy_2d_kernel(unsigned char* __restrict__ dst, size_t dpitch,
                                                      const unsigned char* src, size_t spitch,
                                                      size_t row_elems, size_t rows) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t total = row_elems * rows;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        size_t r = i / row_elems, c = i - r * row_elems;
        *reinterpret_cast<V*>(dst + r * dpitch + c * sizeof(V)) =
            *reinterpret_cast<const V*>(src + r * spitch + c * sizeof(V));
    }
}

static int launch_copy_2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t row_bytes, size_t rows,
                          cudaStream_t st) {
    if (row_bytes == 0 || rows == 0) return PIMB200_OK;
    if (dpitch == row_bytes && spitch == row_bytes) {
        PIMB200_CUDA_TRY(cudaMemcpyAsync(dst, src, row_bytes * rows, cudaMemcpyDeviceToDevice, st));
        return PIMB200_OK;
    }
    unsigned char* d = static_cast<unsigned char*>(dst);
    const unsigned char* s = static_cast<const unsigned char*>(src);
    const uintptr_t bits = reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(s) | dpitch | spitch | row_bytes;
    const size_t total_bytes = row_bytes * rows;
    auto grid_for = [](size_t elems) {
        size_t g = (elems + 255) / 256;
        return (unsigned)(g > 148 * 16 ? 148 * 16 : (g ? g : 1));
    };
    if ((bits & 15) == 0)
        return cuda_status(launch_pdl(copy_2d_kernel<uint4>, dim3(grid_for(total_bytes / 16)), dim3(256), 0, st, d, dpitch, s, spitch,
                                      row_bytes / 16, rows));
    else if ((bits & 3) == 0)
        copy_2d_kernel<uint32_t><<<grid_for(total_bytes / 4), 256, 0, st>>>(d, dpitch, s, spitch, row_bytes / 4, rows);
    else if ((bits & 1) == 0)
        copy_2d_kernel<uint16_t><<<grid_for(total_bytes / 2), 256, 0, st>>>(d, dpitch, s, spitch, row_bytes / 2, rows);
    else
        copy_2d_kernel<uint8_t><<<grid_for(total_bytes), 256, 0, st>>>(d, dpitch, s, spitch, row_bytes, rows);
    return launch_status();
}

// =============================================================================================
// SIMT GEMM:  Y[j,n] = act(sum_k X[j,k] W[n,k] + b[n]) — any shape, any alignment, exact fp32 products and sums.
// 64x64 output tile, 32-deep k slab, 256 threads with a 4x4 register tile each.  The A/B switch of the tensor-core kernels.
// =============================================================================================
template <bool OUT_F32>
__global__ void __launch_bounds__(256) gemm_wx_simt_kernel(const __half* __restrict__ W, const __half* __restrict__ X,
                                                           const __half* __restrict__ bias, void* __restrict__ Yv,
                                                           int N, int K, int J, int ldx, int ldy, int act) {
    constexpr int BN = 64, BJ = 64, BK = 32;
    __shared__ __align__(16) float Ws[BK][BN + 4];
    __shared__ __align__(16) float Xs[BK][BJ + 4];
    const int n0 = blockIdx.x * BN, j0 = blockIdx.y * BJ;
    const int tn = threadIdx.x & 15, tj = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;

    const int lrow = threadIdx.x >> 2;        // 0..63: tile row this thread loads
    const int lk = (threadIdx.x & 3) * 8;     // 0,8,16,24: first k of its 8-wide slice
    for (int kb = 0; kb < K; kb += BK) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int k = kb + lk + e;
            const int n = n0 + lrow, j = j0 + lrow;
            Ws[lk + e][lrow] = (n < N && k < K) ? __half2float(W[(size_t)n * K + k]) : 0.f;
            Xs[lk + e][lrow] = (j < J && k < K) ? __half2float(X[(size_t)j * ldx + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 wv = *reinterpret_cast<const float4*>(&Ws[kk][tn * 4]);
            const float4 xv = *reinterpret_cast<const float4*>(&Xs[kk][tj * 4]);
            const float w4[4] = {wv.x, wv.y, wv.z, wv.w};
            const float x4[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(x4[a], w4[b], acc[a][b]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int j = j0 + tj * 4 + a;
        if (j >= J) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int n = n0 + tn * 4 + b;
            if (n >= N) continue;
            float v = acc[a][b] + (bias ? __half2float(bias[n]) : 0.f);
            if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
            if (OUT_F32)
                static_cast<float*>(Yv)[(size_t)j * ldy + n] = v;
            else
                static_cast<__half*>(Yv)[(size_t)j * ldy + n] = __float2half_rn(v);
        }
    }
}

int launch_gemm_wx_simt(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx,
                        int ldy, int act, int y_is_f32, cudaStream_t st) {
    dim3 grid(ceil_div(N, 64), ceil_div(J, 64));
    if (y_is_f32)
        gemm_wx_simt_kernel<true><<<grid, 256, 0, st>>>(W, X, bias, Y, N, K, J, ldx, ldy, act);
    else
        gemm_wx_simt_kernel<false><<<grid, 256, 0, st>>>(W, X, bias, Y, N, K, J, ldx, ldy, act);
    return launch_status();
}

// =============================================================================================
// Ragged dense contraction: any shape, any alignment (K not a multiple of 8, rows off 16-byte boundaries), where neither TMA
// nor 16-byte loads apply.  64 x 64 tiles by mma.sync, 64-deep slabs read with 2-byte loads along the rows (64 bytes per warp
// and load), the next slab's loads in flight during this one's products.  The SIMT kernel above took 72 us for 517 rows of
// 1280 x 761: eight strided 2-byte loads per thread and slab, nothing in flight meanwhile, and FMAs.
// =============================================================================================
template <bool OUT_F32>
__global__ void __launch_bounds__(256) gemm_wx_ragged_kernel(const __half* __restrict__ W, const __half* __restrict__ X,
                                                             const __half* __restrict__ bias, void* __restrict__ Yv, int N, int K,
                                                             int J, int ldx, int ldy, int act) {
    constexpr int T = 64, BK = 64, P = BK + 8;         // pitch of 144 bytes: ldmatrix rows fall in distinct banks
    __shared__ __align__(16) __half ws[2][T][P], xs[2][T][P];
    const int n0 = blockIdx.x * T, j0 = blockIdx.y * T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wn = warp & 3, wj = warp >> 2;           // this warp's 16 weight rows and 32 activation rows
    const unsigned short* Wu = reinterpret_cast<const unsigned short*>(W);
    const unsigned short* Xu = reinterpret_cast<const unsigned short*>(X);
    uint32_t wv[8], xv[8];                             // rows 8 * warp + i of both tiles, columns lane and lane + 32 of the slab
    auto load = [&](int kb) {
        const int k = kb + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int n = n0 + 8 * warp + i, j = j0 + 8 * warp + i;
            const size_t wr = (size_t)n * K + k, xr = (size_t)j * ldx + k;
            uint32_t w0 = 0, w1 = 0, x0 = 0, x1 = 0;
            if (n < N && k < K) w0 = __ldg(Wu + wr);
            if (n < N && k + 32 < K) w1 = __ldg(Wu + wr + 32);
            if (j < J && k < K) x0 = __ldg(Xu + xr);
            if (j < J && k + 32 < K) x1 = __ldg(Xu + xr + 32);
            wv[i] = w0 | w1 << 16;
            xv[i] = x0 | x1 << 16;
        }
    };
    auto store = [&](int b) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            unsigned short* w = reinterpret_cast<unsigned short*>(ws[b][8 * warp + i]) + lane;
            unsigned short* x = reinterpret_cast<unsigned short*>(xs[b][8 * warp + i]) + lane;
            w[0] = (unsigned short)wv[i];
            w[32] = (unsigned short)(wv[i] >> 16);
            x[0] = (unsigned short)xv[i];
            x[32] = (unsigned short)(xv[i] >> 16);
        }
    };
    auto ldm = [](uint32_t (&r)[4], const __half* p) {
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"((uint32_t)__cvta_generic_to_shared(p))
                     : "memory");
    };
    float acc[4][4];
#pragma unroll
    for (int t = 0; t < 4; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    load(0);
    store(0);
    __syncthreads();
    int b = 0;
    for (int kb = 0; kb < K; kb += BK, b ^= 1) {
        if (kb + BK < K) load(kb + BK);
        float slab[4][4];              // summed apart and added in fp32: the tensor unit's own sums are cut off, not rounded
#pragma unroll
        for (int t = 0; t < 4; ++t) slab[t][0] = slab[t][1] = slab[t][2] = slab[t][3] = 0.f;
#pragma unroll
        for (int k = 0; k < BK; k += 16) {
            uint32_t a[4], x[2][4];
            ldm(a, &ws[b][wn * 16 + (lane & 7) + (lane >> 3 & 1) * 8][k + (lane >> 4) * 8]);
#pragma unroll
            for (int p = 0; p < 2; ++p) ldm(x[p], &xs[b][wj * 32 + p * 16 + (lane & 7) + (lane >> 4) * 8][k + (lane >> 3 & 1) * 8]);
#pragma unroll
            for (int t = 0; t < 4; ++t)
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                             : "+f"(slab[t][0]), "+f"(slab[t][1]), "+f"(slab[t][2]), "+f"(slab[t][3])
                             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(x[t >> 1][2 * (t & 1)]), "r"(x[t >> 1][2 * (t & 1) + 1]));
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[t][e] += slab[t][e];
        if (kb + BK < K) store(b ^ 1);                 // (everyone read that buffer before the last barrier)
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = n0 + wn * 16 + (lane >> 2) + (e >> 1) * 8, j = j0 + wj * 32 + t * 8 + 2 * (lane & 3) + (e & 1);
            if (n >= N || j >= J) continue;
            float v = acc[t][e] + (bias ? __half2float(bias[n]) : 0.f);
            if (act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
            if (OUT_F32) static_cast<float*>(Yv)[(size_t)j * ldy + n] = v;
            else static_cast<__half*>(Yv)[(size_t)j * ldy + n] = __float2half_rn(v);
        }
}

int launch_gemm_wx_ragged(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx, int ldy, int act,
                          int y_is_f32, cudaStream_t st) {
    const dim3 grid(ceil_div(N, 64), ceil_div(J, 64));
    if (y_is_f32) gemm_wx_ragged_kernel<true><<<grid, 256, 0, st>>>(W, X, bias, Y, N, K, J, ldx, ldy, act);
    else gemm_wx_ragged_kernel<false><<<grid, 256, 0, st>>>(W, X, bias, Y, N, K, J, ldx, ldy, act);
    return launch_status();
}

}  // namespace pimb200

// =============================================================================================
// C ABI
// =============================================================================================
using namespace pimb200;

extern "C" int pimb200_gemv_mv(const void* W, const void* x, const void* bias, void* y, int N, int K, int act,
                               void* stream) {
    if (!W || !x || !y || N <= 0 || K <= 0) return PIMB200_ERR_BAD_ARG;
    if (act != PIMB200_ACT_NONE && act != PIMB200_ACT_RELU) return PIMB200_ERR_BAD_ARG;
    return launch_gemv_mv(static_cast<const __half*>(W), static_cast<const __half*>(x),
                          static_cast<const __half*>(bias), static_cast<__half*>(y), N, K, act,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int pimb200_gemv_vm(const void* x, const void* A, const void* bias, void* y, int K, int N, int act,
                               void* stream) {
    if (!A || !x || !y || N <= 0 || K <= 0) return PIMB200_ERR_BAD_ARG;
    if (act != PIMB200_ACT_NONE && act != PIMB200_ACT_RELU) return PIMB200_ERR_BAD_ARG;
    return launch_gemv_vm(static_cast<const __half*>(x), static_cast<const __half*>(A),
                          static_cast<const __half*>(bias), static_cast<__half*>(y), K, N, act, true,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int pimb200_bmm_row(const void* x, const void* A, void* y, int k, int n, void* stream) {
    if (!A || !x || !y || n <= 0 || k <= 0) return PIMB200_ERR_BAD_ARG;
    // same kernel as VM without bias; k is a source-sentence length (tens of rows), so no K split
    return launch_gemv_vm(static_cast<const __half*>(x), static_cast<const __half*>(A), nullptr,
                          static_cast<__half*>(y), k, n, PIMB200_ACT_NONE, false, static_cast<cudaStream_t>(stream));
}

extern "C" int pimb200_dot_vv(const void* a, const void* b, void* y, int K, void* stream) {
    if (!a || !b || !y || K <= 0) return PIMB200_ERR_BAD_ARG;
    dot_vv_kernel<<<1, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __half*>(a),
                                                                   static_cast<const __half*>(b),
                                                                   static_cast<__half*>(y), K);
    return launch_status();
}

extern "C" int pimb200_add_f16(const void* A, const void* B, void* C, int m, int n, int broadcast_b, void* stream) {
    if (!A || !B || !C || m <= 0 || n <= 0) return PIMB200_ERR_BAD_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t total = (size_t)m * n;
    if (n % 8 == 0 && aligned16(A) && aligned16(B) && aligned16(C)) {
        size_t total8 = total / 8;
        size_t g = (total8 + 255) / 256;
        unsigned grid = (unsigned)(g > 148 * 8 ? 148 * 8 : g);
        return cuda_status(launch_pdl(add_f16_vec_kernel, dim3(grid), dim3(256), 0, st, static_cast<const uint4*>(A),
                                      static_cast<const uint4*>(B), static_cast<uint4*>(C), total8, n / 8, broadcast_b ? 1 : 0));
    } else {
        size_t g = (total + 255) / 256;
        unsigned grid = (unsigned)(g > 148 * 8 ? 148 * 8 : g);
        add_f16_scalar_kernel<<<grid, 256, 0, st>>>(static_cast<const __half*>(A), static_cast<const __half*>(B),
                                                    static_cast<__half*>(C), total, n, broadcast_b ? 1 : 0);
    }
    return launch_status();
}

extern "C" int pimb200_copy_2d(void* dst, size_t dst_pitch, const void* src, size_t src_pitch, size_t row_bytes,
                               size_t rows, void* stream) {
    if (!dst || !src) return (row_bytes == 0 || rows == 0) ? PIMB200_OK : PIMB200_ERR_BAD_ARG;
    if (dst_pitch < row_bytes || src_pitch < row_bytes) return PIMB200_ERR_BAD_ARG;
    return launch_copy_2d(dst, dst_pitch, src, src_pitch, row_bytes, rows, static_cast<cudaStream_t>(stream));
}

extern "C" int pimb200_cat(void* dst, const void* const* src, const size_t* inner_bytes, int n_src, size_t outer,
                           void* stream) {
    if (!dst || !src || !inner_bytes || n_src <= 0) return PIMB200_ERR_BAD_ARG;
    size_t pitch = 0;
    for (int i = 0; i < n_src; ++i) pitch += inner_bytes[i];
    size_t off = 0;
    for (int i = 0; i < n_src; ++i) {
        if (inner_bytes[i] == 0) continue;  // empty operands are legal in aten::cat
        if (!src[i]) return PIMB200_ERR_BAD_ARG;
        int rc = launch_copy_2d(static_cast<unsigned char*>(dst) + off, pitch, src[i], inner_bytes[i], inner_bytes[i],
                                outer, static_cast<cudaStream_t>(stream));
        if (rc != PIMB200_OK) return rc;
        off += inner_bytes[i];
    }
    return PIMB200_OK;
}
