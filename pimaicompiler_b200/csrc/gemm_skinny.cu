// Batched-stream linear layer for few activation rows:  Y[J, N] = act(X[J, K] . W[N, K]^T + bias[N]),  J <= 32.
//
// This is the batch 8 / 32 form of the batch-1 GEMV (several utterance streams sharing one weight matrix, or the
// branches of a MULTISTREAM node): the arithmetic intensity is J flop per weight byte, far below the ridge, so the
// bound is the one pass over W from HBM, exactly as for the GEMV.  A 128-row tcgen05 tile per CTA leaves most SMs
// without work at N = 4096 (32 CTAs) and costs a fixed pipeline set-up; here every SM streams W instead:
//   * a CTA owns 16 or 32 weight rows (one or two 16-row tiles) and its 8 warps split K between them; with 32 rows
//     (N >= 2048: one CTA per SM at N = 4096) a warp multiplies both tiles by the same X fragments; every load of a
//     group of K blocks is issued before the previous group's products, so 8 KB per warp are in flight;
//   * a warp reads its W rows with 128-bit loads that bypass L1, 8 consecutive k per thread and row, and uses them
//     directly as mma.sync m16n8k16 A fragments: the contraction index is only a summation order, so the k positions
//     a thread holds (k0 + 8t .. k0 + 8t + 7 of rows g and g + 8) are fed as the fragment's "2t, 2t+1, 2t+8, 2t+9"
//     slots of two products, and the B fragment (X, read through L1: it is small and shared by all CTAs) is taken
//     from the same k positions.  No shared-memory staging, no shuffles;
//   * the K-partials meet in shared memory; the CTA's rows x J outputs get bias, activation and the fp16 (or fp32) store.
#include "gemm_rows.cuh"

namespace pimb200 {

namespace {
constexpr int kSkinnyWarps = 8;
constexpr int kSkinnyThreads = kSkinnyWarps * 32;
constexpr int kSkinnyRows = 16;
constexpr int kSkinnyMaxJ = 32;
constexpr int kSkinnyMaxBlockedJ = 256;                     // column-blocked form: at most 8 blocks of 32 rows ...
constexpr int kSkinnyMaxBlockedN = 2048;                    // ... of a matrix of at most 2048 rows ...
constexpr size_t kSkinnyMaxBlockedNK = (size_t)8 << 20;     // ... and 16 MB
constexpr int kSkinnyMaxBlockedCtas = kNumSmB200;           // ... in one wave of CTAs: 3.5 us at 512 x 512, 128 rows (tcgen05
                                                            // 4.1), but 7.9 at 2048 x 512, 160 rows (4.2)

// not volatile: the compiler may move these products freely (volatile asm statements keep their order, which would put every
// block's loads, which are, behind the previous block's products and serialise the HBM round trips)
__device__ __forceinline__ void mma16816(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 bytes of a handle's weights, which no launch writes: may be loaded ahead of a wait
__device__ __forceinline__ uint4 ldg_w(const __half* p) {
    uint4 r;
    asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

struct SkinnyArgs {
    const __half* W;      // [N, K] row-major
    const __half* X;      // [J, ldx]
    const __half* bias;   // [N] or NULL
    void* Y;              // [J, ldy] fp16 or fp32
    int N, K, J, ldx, ldy, act, y_is_f32;
    float* best_v;        // arg max form: [CTAs][J] largest output of the CTA's rows and its index
    int* best_i;
    int fixed;            // 1: no work ahead on the stream writes W (it may be read before that work has ended)
};

// NT: n-tiles of 8 activation rows; MTW: 16-row weight tiles per warp (1 or 2; they share the warp's X fragments).
// The 8 warps of a CTA split K; a warp walks its K range in groups of UB 32-wide blocks, the loads of the next group
// in flight while the current one is multiplied.
// UB: 32-wide K blocks per register buffer.  One is all that a warp has at K <= 512, and leaves room for CTAs of the launches behind
// this one on the same SM (20 rows: 250 registers with buffers of four).
// AHEAD: both buffers are under way before the first product; else the second one is asked for ahead of the first one's products.
// PER_SM: CTAs that an SM has to hold (0: as the compiler likes).  The arguments come by value: as a grid constant they give the
// form of <1, 2, 2, false, 0> other registers and 20 % more time.
template <int NT, int MTW, int UB, bool AHEAD, int PER_SM>
__global__ void __launch_bounds__(kSkinnyThreads, PER_SM) gemm_skinny_kernel(SkinnyArgs a) {
    constexpr int KS = kSkinnyWarps;
    constexpr int ROWS = MTW * kSkinnyRows;
    __shared__ float part[KS][ROWS][NT * 8 + 1];
    pdl_launch_dependents();
    if (!AHEAD || !a.fixed) pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * ROWS;
    const int K = a.K;
    // this warp's K range, in blocks of 32 (whole blocks; the ragged tail is zero-filled)
    const int blocks = (K + 31) >> 5;
    const int per = (blocks + KS - 1) / KS;
    const int b_lo = warp * per, b_hi = min(blocks, b_lo + per);
    const __half* wrow[MTW][2];   // rows past N repeat the last one (never stored)
#pragma unroll
    for (int m = 0; m < MTW; ++m) {
        wrow[m][0] = a.W + (size_t)min(n0 + m * 16 + g, a.N - 1) * K + 8 * t;
        wrow[m][1] = a.W + (size_t)min(n0 + m * 16 + g + 8, a.N - 1) * K + 8 * t;
    }
    const __half* xrow[NT];
    const int j_base = blockIdx.y * kSkinnyMaxJ;               // this CTA's block of up to 32 activation rows
    const int j_rem = a.J - j_base;
#pragma unroll
    for (int j = 0; j < NT; ++j) xrow[j] = a.X + (size_t)(j_base + min(j * 8 + g, j_rem - 1)) * a.ldx + 8 * t;
    float acc[MTW][NT][4];
#pragma unroll
    for (int m = 0; m < MTW; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][j][i] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 wc[UB][MTW][2], xc[UB][NT], wn[UB][MTW][2], xn[UB][NT];
    // K % 8 == 0: a thread's 8 consecutive k are all inside or all outside
    auto inside = [&](int b) { return b < b_hi && b * 32 + 8 * t < K; };
    auto load_w1 = [&](uint4 (&w)[MTW][2], int b) {
#pragma unroll
        for (int m = 0; m < MTW; ++m) {
            w[m][0] = inside(b) ? ld_stream_v4(wrow[m][0] + (size_t)b * 32) : zero;
            w[m][1] = inside(b) ? ld_stream_v4(wrow[m][1] + (size_t)b * 32) : zero;
        }
    };
    auto load_x1 = [&](uint4 (&x)[NT], int b) {
#pragma unroll
        for (int j = 0; j < NT; ++j) x[j] = inside(b) ? ld_v4(xrow[j] + (size_t)b * 32) : zero;
    };
    auto load_w = [&](uint4 (&w)[UB][MTW][2], int b0) {
#pragma unroll
        for (int u = 0; u < UB; ++u) load_w1(w[u], b0 + u);
    };
    auto load_x = [&](uint4 (&x)[UB][NT], int b0) {
#pragma unroll
        for (int u = 0; u < UB; ++u) load_x1(x[u], b0 + u);
    };
    auto multiply = [&](const uint4 (&w)[UB][MTW][2], const uint4 (&x)[UB][NT]) {
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int m = 0; m < MTW; ++m) {
                    // two products per 32-wide block: k positions {0,1 | 2,3} and {4,5 | 6,7} of the thread's eight
                    mma16816(acc[m][j], w[u][m][0].x, w[u][m][1].x, w[u][m][0].y, w[u][m][1].y, x[u][j].x, x[u][j].y);
                    mma16816(acc[m][j], w[u][m][0].z, w[u][m][1].z, w[u][m][0].w, w[u][m][1].w, x[u][j].z, x[u][j].w);
                }
    };
    // two register buffers used alternately (no copies between them: a move would wait for the load it moves)
    if constexpr (AHEAD) {
        if (a.fixed) {             // weights that nobody writes are on their way before the predecessor has ended
            load_w(wc, b_lo);
            load_w(wn, b_lo + UB);
            pdl_wait();
            load_x(xc, b_lo);
            load_x(xn, b_lo + UB);
        } else {
            load_w(wc, b_lo); load_x(xc, b_lo);
            load_w(wn, b_lo + UB); load_x(xn, b_lo + UB);
        }
        for (int b0 = b_lo; b0 < b_hi; b0 += 2 * UB) {
            multiply(wc, xc);
            load_w(wc, b0 + 2 * UB); load_x(xc, b0 + 2 * UB);
            multiply(wn, xn);
            load_w(wn, b0 + 3 * UB); load_x(xn, b0 + 3 * UB);
        }
    } else {
        auto load = [&](uint4 (&w)[UB][MTW][2], uint4 (&x)[UB][NT], int b0) {
#pragma unroll
            for (int u = 0; u < UB; ++u) {
                const int b = b0 + u;
                const bool in = b < b_hi && b * 32 + 8 * t < K;
#pragma unroll
                for (int m = 0; m < MTW; ++m) {
                    w[u][m][0] = in ? ld_stream_v4(wrow[m][0] + (size_t)b * 32) : zero;
                    w[u][m][1] = in ? ld_stream_v4(wrow[m][1] + (size_t)b * 32) : zero;
                }
#pragma unroll
                for (int j = 0; j < NT; ++j) x[u][j] = in ? ld_v4(xrow[j] + (size_t)b * 32) : zero;
            }
        };
        load(wc, xc, b_lo);
        for (int b0 = b_lo; b0 < b_hi; b0 += 2 * UB) {
            load(wn, xn, b0 + UB);
            multiply(wc, xc);
            load(wc, xc, b0 + 2 * UB);
            multiply(wn, xn);
        }
    }
    // accumulator layout: (row g, cols 2t, 2t+1), (row g+8, same cols) of each n-tile
#pragma unroll
    for (int m = 0; m < MTW; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            part[warp][m * 16 + g][j * 8 + 2 * t] = acc[m][j][0];
            part[warp][m * 16 + g][j * 8 + 2 * t + 1] = acc[m][j][1];
            part[warp][m * 16 + g + 8][j * 8 + 2 * t] = acc[m][j][2];
            part[warp][m * 16 + g + 8][j * 8 + 2 * t + 1] = acc[m][j][3];
        }
    __syncthreads();
    // output (activation row j, weight row r): consecutive threads take consecutive weight rows
    for (int i = threadIdx.x; i < ROWS * NT * 8; i += kSkinnyThreads) {
        const int r = i % ROWS, j = i / ROWS;
        const int n = n0 + r;
        if (n >= a.N || j >= j_rem) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < KS; ++w) v += part[w][r][j];
        if (a.bias) v += __half2float(a.bias[n]);
        if (a.act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        if (a.y_is_f32) static_cast<float*>(a.Y)[(size_t)(j_base + j) * a.ldy + n] = v;
        else static_cast<__half*>(a.Y)[(size_t)(j_base + j) * a.ldy + n] = __float2half_rn(v);
    }
}

// One LSTM step of up to 32 sequences in one launch: the products with W_ih and W_hh as one walk over the K blocks of both
// (their eight warps' partial sums meet once), gate math in the epilogue.  A CTA owns 32 packed gate rows = 8 hidden units.
// As two products and a gate kernel a step of 9 sequences (2048 inputs, H = 1024) took 12.8 us, the first 1.1 of each
// kernel in launch and ramp; one launch takes 8.9.  The weights are constants of the handle, so the first group of them is
// loaded before the kernel's predecessor has finished.
// BLOCKS: more than 32 sequences, in blocks of 32 (of their own instance: with the block's start in a register 9..16 sequences of
// 320..768 units took 3..8 % longer)
template <int NT, bool BLOCKS>
__global__ void __launch_bounds__(kSkinnyThreads) lstm_cell_skinny_kernel(const __grid_constant__ RowsCell a) {
    constexpr int KS = kSkinnyWarps, ROWS = 2 * kSkinnyRows, UB = 2;
    __shared__ float part[KS][ROWS][NT * 8 + 1];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * ROWS;                              // 4H is a multiple of 32
    const int j_base = BLOCKS ? blockIdx.y * kSkinnyMaxJ : 0, J = BLOCKS ? min(a.J - j_base, kSkinnyMaxJ) : a.J;   // this CTA's sequences
    const int bx = a.I >> 5, blocks = bx + (a.h0 ? a.H >> 5 : 0);  // 32-wide K blocks of both products
    const int per = (blocks + KS - 1) / KS;
    const int b_lo = min(blocks, warp * per), b_hi = min(blocks, b_lo + per);
    const __half* wi = a.Wx + (size_t)(n0 + g) * a.I + 8 * t;
    const __half* wh = a.Wh + (size_t)(n0 + g) * a.H + 8 * t;
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[m][j][i] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 wc[UB][2][2], xc[UB][NT], wn[UB][2][2], xn[UB][NT];
    auto load_w = [&](uint4 (&w)[UB][2][2], int b0) {
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int b = b0 + u;
            const bool in = b < b_hi, first = b < bx;
            const __half* p = first ? wi + (size_t)b * 32 : wh + (size_t)(b - bx) * 32;
            const size_t row8 = (size_t)8 * (first ? a.I : a.H);
#pragma unroll
            for (int q = 0; q < 4; ++q) w[u][q >> 1][q & 1] = in ? ldg_w(p + q * row8) : zero;   // rows g, g+8, g+16, g+24
        }
    };
    auto load_x = [&](uint4 (&x)[UB][NT], int b0) {
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int b = b0 + u;
            const bool in = b < b_hi, first = b < bx;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int row = j_base + min(j * 8 + g, J - 1);    // rows past J repeat the last one
                const __half* p = first ? a.x + (size_t)row * a.x_ld + b * 32 : a.h0 + (size_t)row * a.H + (b - bx) * 32;
                x[u][j] = in ? ld_v4(p + 8 * t) : zero;
            }
        }
    };
    auto multiply = [&](const uint4 (&w)[UB][2][2], const uint4 (&x)[UB][NT]) {
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    mma16816(acc[m][j], w[u][m][0].x, w[u][m][1].x, w[u][m][0].y, w[u][m][1].y, x[u][j].x, x[u][j].y);
                    mma16816(acc[m][j], w[u][m][0].z, w[u][m][1].z, w[u][m][0].w, w[u][m][1].w, x[u][j].z, x[u][j].w);
                }
    };
    // the CTA's rows of both matrices, 128 to 256 KB, on their way into L2 while the predecessor finishes
    if (BLOCKS && blockIdx.y > 0) {
    } else if (threadIdx.x < 32) prefetch_l2(a.Wx + (size_t)(n0 + lane) * a.I, (uint32_t)a.I * 2);
    else if (threadIdx.x < 64 && a.h0) prefetch_l2(a.Wh + (size_t)(n0 + lane) * a.H, (uint32_t)a.H * 2);
    load_w(wc, b_lo);
    pdl_wait();
    load_x(xc, b_lo);
    for (int b0 = b_lo; b0 < b_hi; b0 += 2 * UB) {
        load_w(wn, b0 + UB); load_x(xn, b0 + UB);
        multiply(wc, xc);
        load_w(wc, b0 + 2 * UB); load_x(xc, b0 + 2 * UB);
        multiply(wn, xn);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[warp][m * 16 + g + (e >> 1) * 8][j * 8 + 2 * t + (e & 1)] = acc[m][j][e];
    __syncthreads();
    const int ul = threadIdx.x & 7, u = (n0 >> 2) + ul;            // a thread per (sequence, unit)
    for (int j = threadIdx.x >> 3; j < J; j += kSkinnyThreads / 8) {
        const size_t row = j_base + j;
        const float4 b4 = *reinterpret_cast<const float4*>(a.bias + (size_t)u * 4);
        float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < KS; ++w)
#pragma unroll
            for (int q = 0; q < 4; ++q) z[q] += part[w][ul * 4 + q][j];
        const float cprev = a.c0 ? __half2float(a.c0[row * a.H + u]) : 0.f;
        const float cnew = sigmoidf_(z[1] + b4.y) * cprev + sigmoidf_(z[0] + b4.x) * tanhf_(z[2] + b4.z);
        const __half hh = __float2half_rn(sigmoidf_(z[3] + b4.w) * tanhf_(cnew));
        a.y[row * a.y_ld + u] = a.res ? __float2half_rn(__half2float(hh) + __half2float(a.res[row * a.res_ld + u])) : hh;
        if (a.hn) a.hn[row * a.H + u] = hh;
        if (a.cn) a.cn[row * a.H + u] = __float2half_rn(cnew);
    }
}

// Many weight rows (N >= 16384: the vocabulary projection of a batched decode step) and 9..32 activation rows: one
// warp per 16-row tile over the whole of K, no K split, so nothing is folded through shared memory and no barrier
// follows the start.  Read straight from global memory the X fragments would cost as many load slots and registers as
// W itself; here the CTA copies X into shared memory once (cp.async; odd rows stored with their 16-byte chunks swapped
// across 64 bytes, so a quarter-warp's 128-bit reads - two rows x 64 bytes - fall in distinct banks) and its 8 warps
// walk tiles of a persistent grid, two register buffers of W loads in flight per warp.
// Several independent products in ONE launch (the branches of a MULTISTREAM node: a few activation rows against
// different weight matrices): blockIdx.z selects the problem, blockIdx.y its block of 32 activation rows, blockIdx.x its
// 16-row weight tile; CTAs past a problem's extent leave at once.  Same arithmetic as gemm_skinny_kernel<NT, 1>.
constexpr int kGroupedMax = 8;
struct GroupedArgs {
    SkinnyArgs p[kGroupedMax];
};

template <int NT>
__global__ void __launch_bounds__(kSkinnyThreads) gemm_skinny_grouped_kernel(const __grid_constant__ GroupedArgs ga) {
    constexpr int KS = kSkinnyWarps;
    constexpr int UB = 4;
    __shared__ float part[KS][kSkinnyRows][NT * 8 + 1];
    pdl_launch_dependents();
    pdl_wait();
    const SkinnyArgs& a = ga.p[blockIdx.z];
    const int n0 = blockIdx.x * kSkinnyRows;
    const int j_base = blockIdx.y * kSkinnyMaxJ;
    if (n0 >= a.N || j_base >= a.J) return;                    // CTA-uniform
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int K = a.K;
    const int blocks = (K + 31) >> 5;
    const int per = (blocks + KS - 1) / KS;
    const int b_lo = warp * per, b_hi = min(blocks, b_lo + per);
    const __half* w_lo = a.W + (size_t)min(n0 + g, a.N - 1) * K + 8 * t;
    const __half* w_hi = a.W + (size_t)min(n0 + g + 8, a.N - 1) * K + 8 * t;
    const int j_rem = a.J - j_base;
    const __half* xrow[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) xrow[j] = a.X + (size_t)(j_base + min(j * 8 + g, j_rem - 1)) * a.ldx + 8 * t;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 wc[UB][2], xc[UB][NT], wn[UB][2], xn[UB][NT];
    auto load_group = [&](uint4 (&w)[UB][2], uint4 (&x)[UB][NT], int b0) {
#pragma unroll
        for (int u = 0; u < UB; ++u) {
            const int b = b0 + u;
            const bool in = b < b_hi && b * 32 + 8 * t < K;
            w[u][0] = in ? ld_stream_v4(w_lo + (size_t)b * 32) : zero;
            w[u][1] = in ? ld_stream_v4(w_hi + (size_t)b * 32) : zero;
#pragma unroll
            for (int j = 0; j < NT; ++j) x[u][j] = in ? ld_v4(xrow[j] + (size_t)b * 32) : zero;
        }
    };
    auto multiply = [&](const uint4 (&w)[UB][2], const uint4 (&x)[UB][NT]) {
#pragma unroll
        for (int u = 0; u < UB; ++u)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                mma16816(acc[j], w[u][0].x, w[u][1].x, w[u][0].y, w[u][1].y, x[u][j].x, x[u][j].y);
                mma16816(acc[j], w[u][0].z, w[u][1].z, w[u][0].w, w[u][1].w, x[u][j].z, x[u][j].w);
            }
    };
    load_group(wc, xc, b_lo);
    for (int b0 = b_lo; b0 < b_hi; b0 += 2 * UB) {
        load_group(wn, xn, b0 + UB);
        multiply(wc, xc);
        load_group(wc, xc, b0 + 2 * UB);
        multiply(wn, xn);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        part[warp][g][j * 8 + 2 * t] = acc[j][0];
        part[warp][g][j * 8 + 2 * t + 1] = acc[j][1];
        part[warp][g + 8][j * 8 + 2 * t] = acc[j][2];
        part[warp][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSkinnyRows * NT * 8; i += kSkinnyThreads) {
        const int r = i % kSkinnyRows, j = i / kSkinnyRows;
        const int n = n0 + r;
        if (n >= a.N || j >= j_rem) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < KS; ++w) v += part[w][r][j];
        if (a.bias) v += __half2float(a.bias[n]);
        if (a.act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
        if (a.y_is_f32) static_cast<float*>(a.Y)[(size_t)(j_base + j) * a.ldy + n] = v;
        else static_cast<__half*>(a.Y)[(size_t)(j_base + j) * a.ldy + n] = __float2half_rn(v);
    }
}

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
    uint4 r;
    asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(addr));
    return r;
}

// FULL: K a multiple of 128 (no partial group of K blocks).  ARGMAX: nothing is stored but, per CTA and activation row, the
// largest output (rounded to fp16, as it would be stored) and the lowest index that has it.
template <int NT, bool FULL, bool ARGMAX>
__global__ void __launch_bounds__(kSkinnyThreads, 2) gemm_skinny_rows_kernel(SkinnyArgs a, int tiles) {
    constexpr int UB = 4;                                            // 32-wide K blocks per register buffer
    extern __shared__ __align__(16) unsigned char sk_smem[];
    pdl_launch_dependents();
    if (!a.fixed) pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int K = a.K;                                               // K % 64 == 0 (checked by the launcher)
    const int xs = K * 2;                                            // bytes per X row, a multiple of 128
    const int blocks = K >> 5;
    const int gpt = (blocks + UB - 1) / UB;                          // groups of K blocks per tile
    auto copy_x = [&] {
        const int chunks = K >> 3;                                   // 16-byte chunks per row
        for (int row = warp; row < NT * 8; row += kSkinnyWarps) {
            const __half* src = a.X + (size_t)min(row, a.J - 1) * a.ldx;   // rows past J repeat the last one
            unsigned char* dst = sk_smem + (size_t)row * xs;
            const int flip = (row & 1) << 2;
            for (int c = lane; c < chunks; c += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + ((c ^ flip) << 4))),
                             "l"(src + c * 8) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // tile i of the launch belongs to CTA i % gridDim.x, warp (i / gridDim.x) % 8; a warp walks its tiles as one stream of
    // (tile, group) pairs, so the loads of a tile's first group are in flight during the previous tile's last products
    const int stride = kSkinnyWarps * gridDim.x;
    uint4 w0[UB][2], w1[UB][2];
    auto load_group = [&](uint4 (&w)[UB][2], int tile, int grp) {
        if (tile >= tiles) return;                                   // warp-uniform
        const int n0 = tile * kSkinnyRows;
        const __half* p_lo = a.W + (size_t)min(n0 + g, a.N - 1) * K + 8 * t + grp * (UB * 32);   // rows past N repeat the last
        const __half* p_hi = a.W + (size_t)min(n0 + g + 8, a.N - 1) * K + 8 * t + grp * (UB * 32);
#pragma unroll
        for (int u = 0; u < UB; ++u)
            if (FULL || grp * UB + u < blocks) {
                w[u][0] = ld_stream_v4(p_lo + u * 32);
                w[u][1] = ld_stream_v4(p_hi + u * 32);
            }
    };
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const uint32_t xaddr = (uint32_t)__cvta_generic_to_shared(sk_smem) + (uint32_t)(g * xs + t * 16);
    const int s1 = g & 1;                                            // odd rows: 64-byte halves of a 128-byte pair swapped
    float top[NT][2];
    int at[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        top[j][0] = top[j][1] = -INFINITY;
        at[j][0] = at[j][1] = 0x7fffffff;
    }
    auto step = [&](const uint4 (&w)[UB][2], int tile, int grp) {
#pragma unroll
        for (int u = 0; u < UB; ++u)
            if (FULL || grp * UB + u < blocks) {
                const uint32_t xb = xaddr + (uint32_t)(((grp * UB + u) ^ s1) << 6);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint4 xv = lds_v4(xb + (uint32_t)(j * 8 * xs));
                    mma16816(acc[j], w[u][0].x, w[u][1].x, w[u][0].y, w[u][1].y, xv.x, xv.y);
                    mma16816(acc[j], w[u][0].z, w[u][1].z, w[u][0].w, w[u][1].w, xv.z, xv.w);
                }
            }
        if (grp != gpt - 1) return;
        // the tile is complete.  Accumulator layout: (row g, cols 2t, 2t+1), (row g+8, same cols) of each n-tile
        const int n0 = tile * kSkinnyRows;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + g + 8 * h;
            const float bv = (a.bias && n < a.N) ? __half2float(a.bias[n]) : 0.f;
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = j * 8 + 2 * t + e;
                    float v = acc[j][2 * h + e] + bv;
                    acc[j][2 * h + e] = 0.f;
                    if (n >= a.N || col >= a.J) continue;
                    if (ARGMAX) {   // a lane's rows come in ascending order
                        v = __half2float(__float2half_rn(v));
                        if (v > top[j][e] || (at[j][e] == 0x7fffffff && v == v)) { top[j][e] = v; at[j][e] = n; }
                        continue;
                    }
                    if (a.act == PIMB200_ACT_RELU) v = fmaxf(v, 0.f);
                    if (a.y_is_f32) static_cast<float*>(a.Y)[(size_t)col * a.ldy + n] = v;
                    else static_cast<__half*>(a.Y)[(size_t)col * a.ldy + n] = __float2half_rn(v);
                }
        }
    };
    auto advance = [&](int& tile, int& grp) {
        if (++grp == gpt) { grp = 0; tile += stride; }
    };
    int lt = blockIdx.x + warp * gridDim.x, lg = 0;                  // load cursor
    int ct = lt, cg = 0;                                             // compute cursor
    if (!a.fixed) copy_x();
    load_group(w0, lt, lg); advance(lt, lg);
    if (a.fixed) {                                                   // the weights are on their way before the predecessor has ended
        pdl_wait();
        copy_x();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                                 // reached by every warp, with or without a tile
    while (ct < tiles) {
        load_group(w1, lt, lg); advance(lt, lg);
        step(w0, ct, cg); advance(ct, cg);
        if (ct >= tiles) break;
        load_group(w0, lt, lg); advance(lt, lg);
        step(w1, ct, cg); advance(ct, cg);
    }
    if (ARGMAX) {
        // over the eight lanes that hold other rows of the same columns, then over the warps
        __shared__ float red_v[kSkinnyWarps][NT * 8];
        __shared__ int red_i[kSkinnyWarps][NT * 8];
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, top[j][e], o);
                    const int oi = __shfl_xor_sync(0xffffffffu, at[j][e], o);
                    if (ov > top[j][e] || (ov == top[j][e] && oi < at[j][e])) { top[j][e] = ov; at[j][e] = oi; }
                }
                if (g == 0) {
                    red_v[warp][j * 8 + 2 * t + e] = top[j][e];
                    red_i[warp][j * 8 + 2 * t + e] = at[j][e];
                }
            }
        __syncthreads();
        const int col = threadIdx.x;
        if (col < NT * 8 && col < a.J) {
            float v = red_v[0][col];
            int i = red_i[0][col];
#pragma unroll
            for (int w = 1; w < kSkinnyWarps; ++w)
                if (red_v[w][col] > v || (red_v[w][col] == v && red_i[w][col] < i)) { v = red_v[w][col]; i = red_i[w][col]; }
            a.best_v[(size_t)blockIdx.x * a.J + col] = v;
            a.best_i[(size_t)blockIdx.x * a.J + col] = i;
        }
    }
}

int skinny_rows_grid(int N, size_t smem) {
    const int per_sm = smem <= 110 * 1024 ? 2 : 1;
    return min(ceil_div(ceil_div(N, kSkinnyRows), kSkinnyWarps), kNumSmB200 * per_sm);
}

template <int NT, bool ARGMAX>
int launch_skinny_rows(const SkinnyArgs& a, cudaStream_t st) {
    const size_t smem = (size_t)NT * 8 * a.K * 2;
    if (a.K % 64 != 0 || smem > 200 * 1024) return PIMB200_ERR_UNSUPPORTED;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return PIMB200_ERR_UNSUPPORTED;
    if (!attr_set[dev]) {
        if (cudaFuncSetAttribute(gemm_skinny_rows_kernel<NT, true, ARGMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_skinny_rows_kernel<NT, false, ARGMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
            return PIMB200_ERR_LAUNCH;
        attr_set[dev] = true;
    }
    const int tiles = ceil_div(a.N, kSkinnyRows);
    const dim3 grid(skinny_rows_grid(a.N, smem)), block(kSkinnyThreads);
    if (a.K % 128 == 0) return cuda_status(launch_pdl(gemm_skinny_rows_kernel<NT, true, ARGMAX>, grid, block, smem, st, a, tiles));
    return cuda_status(launch_pdl(gemm_skinny_rows_kernel<NT, false, ARGMAX>, grid, block, smem, st, a, tiles));
}
}  // namespace

// PIMB200_ERR_UNSUPPORTED when the shape is not this kernel's (the caller then takes the tensor-core or SIMT path)
int launch_gemm_wx_skinny(const __half* W, const __half* X, const __half* bias, void* Y, int N, int K, int J, int ldx,
                          int ldy, int act, int y_is_f32, cudaStream_t st, int fixed) {
    if (J < 1 || K % 8 != 0 || ldx % 8 != 0 || !aligned16(W) || !aligned16(X)) return PIMB200_ERR_UNSUPPORTED;
    // More than 32 activation rows run as column blocks of 32 (grid.y) when the weight matrix is small: W then comes
    // from L2 for all but the first block, and a matrix of a few 128-row tiles would leave most SMs of the tcgen05
    // kernel's grid without work (a Transformer layer's 512 x 512 projections for 128 sequences: 4 tiles).
    if (J > kSkinnyMaxJ && (J > kSkinnyMaxBlockedJ || N > kSkinnyMaxBlockedN || (size_t)N * K > kSkinnyMaxBlockedNK ||
                            ceil_div(N, kSkinnyRows) * ceil_div(J, kSkinnyMaxJ) > kSkinnyMaxBlockedCtas))
        return PIMB200_ERR_UNSUPPORTED;
    SkinnyArgs a{W, X, bias, Y, N, K, J, ldx, ldy, act, y_is_f32, nullptr, nullptr, fixed};
    const int nt = J > kSkinnyMaxJ ? 4 : ceil_div(J, 8);
    const int jblocks = ceil_div(J, kSkinnyMaxJ);
    if (nt >= 2 && N >= 16384 && jblocks == 1) {
        // a warp per row tile with X in shared memory, when the CTA's copy of X fits
        const int rc = nt == 2 ? launch_skinny_rows<2, false>(a, st) : nt == 3 ? launch_skinny_rows<3, false>(a, st)
                                                                    : launch_skinny_rows<4, false>(a, st);
        if (rc != PIMB200_ERR_UNSUPPORTED) return rc;
    }
    const bool wide = N >= 2048;
    const dim3 grid(ceil_div(N, wide ? 2 * kSkinnyRows : kSkinnyRows), jblocks);
    // K blocks per buffer (two buffers per warp).  16 weight rows: as few as hold the warp's share of K, at most four.  32: one at
    // K <= 512, and where a second CTA per SM has work (8192 x 2048, 1 / 20 / 32 rows: 5.1 / 7.4 / 9.0 us with two, 3.9 / 6.4 / 8.0
    // with one), else two (4096 x 1024, 20 rows: 2.8 us, 4.0 with one).
#define PIMB200_ROW(MTW, UB, AHEAD, PER_SM) \
    {gemm_skinny_kernel<1, MTW, UB, AHEAD, PER_SM>, gemm_skinny_kernel<2, MTW, UB, AHEAD, PER_SM>, \
     gemm_skinny_kernel<3, MTW, UB, AHEAD, PER_SM>, gemm_skinny_kernel<4, MTW, UB, AHEAD, PER_SM>}
    static void (*const narrow[3][4])(SkinnyArgs) = {PIMB200_ROW(1, 1, true, 2), PIMB200_ROW(1, 2, true, 1), PIMB200_ROW(1, 4, true, 1)};
    static void (*const broad[2][4])(SkinnyArgs) = {PIMB200_ROW(2, 1, true, 2), PIMB200_ROW(2, 2, true, 1)};
#undef PIMB200_ROW
    const int ctas = grid.x * grid.y;
    void (*kernel)(SkinnyArgs);
    if (wide) {
        const bool one_wave = ctas <= kNumSmB200;
        // up to 8 rows whose weights are loaded ahead of the wait: two in any number of waves (32320 x 1024, 2 rows: 11.9, 13.4 with one)
        kernel = broad[K > 512 ? one_wave || (nt == 1 && fixed) : one_wave && nt == 3][nt - 1];
        // Behind the wait, up to 16 rows and more CTAs than two per SM hold: as many CTAs per SM as registers allow, the buffers one
        // after the other (12000 x 768, 2 / 12 rows: 5.7 / 6.4 us, 6.4 / 8.2 with both under way; 16384 x 512, 2 rows: 5.1 / 5.5; 24000 x
        // 1024: 9.9 / 10.5; 32320 x 1024, weights in L2: 8.5 / 9.7).  17..24 rows in more than one wave: the buffers one after the other
        // (8192 x 1024: 5.9 / 6.5)
        if (!fixed && nt <= 2 && ctas > 2 * kNumSmB200)
            kernel = nt == 2 ? gemm_skinny_kernel<2, 2, 1, false, 0> : K <= 512 ? gemm_skinny_kernel<1, 2, 1, false, 0> : gemm_skinny_kernel<1, 2, 2, false, 0>;
        else if (!fixed && nt == 3 && !one_wave) kernel = gemm_skinny_kernel<3, 2, 1, false, 2>;
    } else {
        int form = K <= 512 ? 0 : K <= 1024 ? 1 : 2;
        // behind the wait: 17..24 rows with one (512 x 768: 3.1 us, 3.3 with two), and 9..24 rows of more than 32 CTAs at K > 768 with four
        // (1024 x 1024, 16 / 24 rows: 2.9 / 3.3, 3.1 / 3.7 with fewer)
        if (!fixed && nt == 3 && K <= 1024) form = 0;
        if (!fixed && (nt == 2 || nt == 3) && K > 768 && grid.x > 32) form = 2;
        kernel = narrow[form][nt - 1];
    }
    const cudaError_t rc = launch_pdl(kernel, grid, dim3(kSkinnyThreads), 0, st, a);
    return cuda_status(rc);
}

int launch_lstm_cell_skinny(const RowsCell& c, cudaStream_t st) {
    if (c.J < 1 || c.J > 65535 * kSkinnyMaxJ || c.I % 32 != 0 || c.H % 32 != 0 || c.x_ld % 8 != 0 || !aligned16(c.x) || (c.h0 && !aligned16(c.h0)))
        return PIMB200_ERR_UNSUPPORTED;
    const dim3 grid(4 * c.H / (2 * kSkinnyRows), ceil_div(c.J, kSkinnyMaxJ)), block(kSkinnyThreads);
    if (grid.y > 1) return cuda_status(launch_pdl(lstm_cell_skinny_kernel<4, true>, grid, block, 0, st, c));
    switch (ceil_div(c.J, 8)) {
        case 1: return cuda_status(launch_pdl(lstm_cell_skinny_kernel<1, false>, grid, block, 0, st, c));
        case 2: return cuda_status(launch_pdl(lstm_cell_skinny_kernel<2, false>, grid, block, 0, st, c));
        case 3: return cuda_status(launch_pdl(lstm_cell_skinny_kernel<3, false>, grid, block, 0, st, c));
        default: return cuda_status(launch_pdl(lstm_cell_skinny_kernel<4, false>, grid, block, 0, st, c));
    }
}

// The arg max form for up to 32 activation rows: best_v / best_i [*parts][J]
int launch_skinny_argmax(const __half* W, const __half* X, const __half* bias, float* best_v, int* best_i, int* parts, int N, int K,
                         int J, int ldx, cudaStream_t st) {
    if (J < 1 || J > kSkinnyMaxJ || K % 64 != 0 || ldx % 8 != 0 || !aligned16(W) || !aligned16(X)) return PIMB200_ERR_UNSUPPORTED;
    const SkinnyArgs a{W, X, bias, nullptr, N, K, J, ldx, 0, PIMB200_ACT_NONE, 0, best_v, best_i, 0};
    const int nt = ceil_div(J, 8);
    *parts = skinny_rows_grid(N, (size_t)nt * 8 * K * 2);
    switch (nt) {
        case 1: return launch_skinny_rows<1, true>(a, st);
        case 2: return launch_skinny_rows<2, true>(a, st);
        case 3: return launch_skinny_rows<3, true>(a, st);
        default: return launch_skinny_rows<4, true>(a, st);
    }
}

// Up to 8 problems in one launch; PIMB200_ERR_UNSUPPORTED when one of them is not a shape of the few-row kernels (the
// caller then launches them one by one)
int launch_gemm_wx_grouped(const GemmProblem* pr, int n, cudaStream_t st) {
    if (n < 1 || n > kGroupedMax) return PIMB200_ERR_UNSUPPORTED;
    GroupedArgs ga;
    int max_tiles = 0, max_jb = 0, max_j = 0;
    for (int i = 0; i < n; ++i) {
        const GemmProblem& q = pr[i];
        if (q.J < 1 || q.J > kSkinnyMaxBlockedJ || q.K % 8 != 0 || q.ldx % 8 != 0 || !aligned16(q.W) || !aligned16(q.X))
            return PIMB200_ERR_UNSUPPORTED;
        if (q.J > kSkinnyMaxJ && (q.N > kSkinnyMaxBlockedN || (size_t)q.N * q.K > kSkinnyMaxBlockedNK)) return PIMB200_ERR_UNSUPPORTED;
        ga.p[i] = SkinnyArgs{q.W, q.X, q.bias, q.Y, q.N, q.K, q.J, q.ldx, q.ldy, q.act, q.y_is_f32, nullptr, nullptr, 0};
        max_tiles = max(max_tiles, ceil_div(q.N, kSkinnyRows));
        max_jb = max(max_jb, ceil_div(q.J, kSkinnyMaxJ));
        max_j = max(max_j, min(q.J, kSkinnyMaxJ));
    }
    for (int i = n; i < kGroupedMax; ++i) ga.p[i] = SkinnyArgs{};
    const dim3 grid(max_tiles, max_jb, n);
    cudaError_t rc = cudaSuccess;
    switch (ceil_div(max_j, 8)) {
        case 1: rc = launch_pdl(gemm_skinny_grouped_kernel<1>, grid, dim3(kSkinnyThreads), 0, st, ga); break;
        case 2: rc = launch_pdl(gemm_skinny_grouped_kernel<2>, grid, dim3(kSkinnyThreads), 0, st, ga); break;
        case 3: rc = launch_pdl(gemm_skinny_grouped_kernel<3>, grid, dim3(kSkinnyThreads), 0, st, ga); break;
        default: rc = launch_pdl(gemm_skinny_grouped_kernel<4>, grid, dim3(kSkinnyThreads), 0, st, ga); break;
    }
    return cuda_status(rc);
}

}  // namespace pimb200
