// The recurrence of one LSTM layer for up to 16 lock-step sequences, or of two stacked layers as a wavefront for up to 8,
// in one cooperative launch of all T steps (H a multiple of 16 up to 1024).
//
// A step's time is the latency of its chain: product -> partial sums -> gates -> all-to-all exchange of the new hidden
// states through L2.  The exchange was two thirds of it (3.7 of 5.0 thousand cycles): records, a release that waits for
// them, a flag, polling, an acquire, and a bulk copy into shared memory, three L2 round trips and four CTA barriers.  Here
// the records validate themselves and travel straight into the registers that multiply them:
//   * a CTA owns 8 hidden units (32 gate rows).  Its record of a sequence is the 8 new hidden values, 16 bytes.  A record
//     that has not arrived holds a sentinel, the fp16 pattern 0xffff, which no hidden value has (NaN is stored as 0x7fff,
//     those of the initial states too);
//     every 32-bit word is checked, so nothing is assumed about a record arriving in one piece.  There is no flag and no
//     release: one L2 trip from the writer's store to the reader's load;
//   * four buffers are used in turn.  At step s a warp of its own writes sentinels into the CTA's records of buffer
//     (s + 2) % 4 and fences; the next step's barrier orders that before the CTA publishes step s + 1.  A reader looks at that
//     buffer only after it has read the same CTA's record of step s + 1, and its old contents (step s - 2) have been read
//     by everyone, since every CTA has published step s - 1.  A launch starts on buffers that the previous launch of the
//     handle has filled with sentinels (two sets, alternating; in a captured call a fill of its own does that);
//   * the eight warps split K into blocks of 32 columns, and a lane polls exactly the records that are its B fragments: the
//     contraction index is only a summation order, so lane (sequence g, t) of a block takes units 8t .. 8t+7 of it as one
//     16-byte record, and W_hh lies in registers (or shared memory) in the same order.  No staging, no barrier between
//     exchange and product: a warp starts multiplying when its own records are there;
//   * one handover per step: the product warps store their partial sums (double-buffered), arrive at the step's named
//     barrier and go on to the next step's records; four gate warps wait there.  Eight lanes hold the units of one record
//     and store it as four 32-bit words.
// How far a product warp can be ahead of its gates: past its look at the records of step s + 1, it holds a record of a CTA
// that published step s + 1, so all product warps of that CTA held this CTA's records of step s, so the gates here have left
// the barrier of step s.  While they wait at that of step s + 1, a product warp is thus at most polling in step s + 3:
// partial sums of two steps suffice, and four barriers, used in turn, never mix two steps' arrivals.
// Wavefront: layer B runs two steps behind layer A (see DirectArgs).  Its input product W_ih(B) . h_A of the next step is
// made from the registers that hold h_A, while the gates work and the records are on their way, and stays in the
// accumulators that W_hh(B) . h_B then continues.
// Measured at H = 1024, one sequence: 2.80 -> 1.30 us per step for one layer, 2.72 -> 1.81 for a wavefront.
// What the memory model gives and what is observed: a record's words are relaxed stores and loads, and every word is looked at,
// so nothing hangs on their order.  That a lane which has seen a CTA's record of step s + 1 finds that CTA's sentinels of
// buffer (s + 2) % 4, fenced ahead of it, and not the older record, rests on its own two loads staying in order: they are
// relaxed loads of different addresses, ordered by control flow only (an acquire would invalidate L1 and cost 380 cycles a
// step).  An SM issues them in order and L2 answers from one copy; no wrong value has been seen.
// Every wait is bounded; a CTA that gives up raises the status word, and the others, polling, see it.  Giving up keeps the
// handover exact, or the gates would wait at a barrier for ever: a product warp that gives up in step s notes the step
// (dead_step keeps the smallest), arrives at that step's barrier and leaves.  The gates pass the barrier of the smallest
// such step, where every product warp has arrived once, and leave behind it without publishing: what the others hold is
// thus always the sum of all product warps, and the bound on who can be where, above, holds while CTAs give up too.
// A warp that gives up in a later step arrives at a barrier that nobody waits for.
#include "lstm_direct.cuh"

namespace pimb200 {
namespace {

constexpr int kWarps = 8;                       // product warps, two warpgroups
constexpr int kGateWarps = 4;                   // 128 cells: 8 units x 16 slots.  They give registers to the product warps
                                                // (168 a thread at launch: 8 x 216 + 4 x 72 = 12 x 168)
constexpr int kThreads = (kWarps + kGateWarps) * 32;
constexpr int kMaxBlocks = 4;                   // K blocks of 32 per warp: H <= 1024
constexpr int kNotDead = 0x7fffffff;

__device__ __forceinline__ void mma_16816(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_relaxed(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool arrived(const uint4& v) { return max(max(v.x, v.y), max(v.z, v.w)) != 0xffffffffu; }

// eight columns x 32 rows: w[m][0 / 1] = W[row 16m + g / 16m + g + 8][the lane's eight k], x = the lane's record
__device__ __forceinline__ void multiply(float (&acc)[2][4], const uint4 (&w)[2][2], const uint4& x) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        mma_16816(acc[m], w[m][0].x, w[m][1].x, w[m][0].y, w[m][1].y, x.x, x.y);
        mma_16816(acc[m], w[m][0].z, w[m][1].z, w[m][0].w, w[m][1].w, x.z, x.w);
    }
}

// LAYERS 1 or 2; NT tiles of 8 sequences (2 only with one layer)
template <int LAYERS, int NT>
__global__ void __launch_bounds__(kThreads, 1) lstm_direct_kernel(const __grid_constant__ DirectArgs a) {
    constexpr int ZP = NT * 8 + 1;                               // odd pitch: the gate lanes' 16-byte reads hit distinct banks
    constexpr int ZL = 8 * ZP * 4;                               // floats of one warp's and layer's partial sums: [unit][ZP][gate]
    constexpr int ZW = LAYERS * ZL, ZBUF = kWarps * ZW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* zpart = reinterpret_cast<float*>(smem_raw);           // [2][warp][layer][unit][ZP][gate]
    uint4* wib = reinterpret_cast<uint4*>(zpart + 2 * ZBUF);      // W_ih(B): [block][m][row half][lane]
    __shared__ int dead_step;                                    // the first step in which a wait gave up
    const int H = a.H, T = a.T, B = a.B;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int n_cta = gridDim.x, cta = blockIdx.x, u0 = cta * 8;
    const int blocks = (n_cta + 3) >> 2;                         // K blocks of four octets
    const int slots = LAYERS * B;
    // An odd number of records is padded with a copy of the last one: stores of half a 32-byte sector cost L2 more (one
    // sequence: 1.49 -> 1.41 us per step).  Records of a CTA in a buffer: 64 to 256 bytes (with less, one 128-byte line takes
    // the stores of too many CTAs).
    const int padded = (slots + 1) & ~1;
    const int stride = slots <= 4 ? 4 : (slots <= 8 ? 8 : 16);
    const size_t buf = (size_t)n_cta * stride;
    if (tid == 0) dead_step = kNotDead;
    for (int i = tid; i < 2 * ZBUF; i += kThreads) zpart[i] = 0.f;   // (warps without a block never write theirs)
    for (size_t i = (size_t)cta * kThreads + tid; i < kDirectSetWords; i += (size_t)n_cta * kThreads)
        a.other_set[i] = make_uint4(~0u, ~0u, ~0u, ~0u);

    if (LAYERS == 2)
        for (int i = tid; i < blocks * 4 * 32; i += kThreads) {
            const int ln = i & 31, q = (i >> 5) & 3, o = 4 * (i >> 7) + (ln & 3);
            wib[i] = o < n_cta ? __ldg(reinterpret_cast<const uint4*>(a.WihB + (size_t)(u0 * 4 + q * 8 + (ln >> 2)) * H + 8 * o)) : make_uint4(0u, 0u, 0u, 0u);
        }
    const int last = T - 1 + (LAYERS == 2 ? 2 : 0);
    __syncthreads();

    if (warp >= kWarps) {
        // ================================ gate warps ================================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;" ::: "memory");
        // cell of this thread: unit gt % 8 of slot gt / 8 (layer-major); the pad repeats the last slot's
        const int gt = tid - kWarps * 32, gu = gt & 7, slot = gt >> 3, u = u0 + gu;
        const bool live = slot < padded, own = slot < slots, has_cells = (warp - kWarps) * 4 < padded;
        const int cell = own ? slot : slots - 1, layer = LAYERS == 2 && cell >= B ? 1 : 0, gn = cell - layer * B;
        const bool sweeps = warp == kWarps + kGateWarps - 1;     // writes the sentinels
        float c = 0.f;
        __half hh = __float2half_rn(0.f);
        float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f), gx = bias4;
        const float* gp = a.G;
        long g_step = 0;
        if (live) {
            if (a.c0[layer]) c = __half2float(a.c0[layer][(size_t)gn * H + u]);
            // (through fp32, which leaves a NaN as 0x7fff: layer B's first records are the caller's own bits otherwise)
            if (a.h0[layer]) hh = __float2half_rn(__half2float(a.h0[layer][(size_t)gn * H + u]));
            bias4 = *reinterpret_cast<const float4*>(a.bias[layer] + (size_t)u * 4);
            if (layer == 0) {
                gp = a.G + (size_t)(a.reverse ? T - 1 : 0) * a.g_tstride + (size_t)gn * a.g_bstride + (size_t)u * 4;
                g_step = a.reverse ? -a.g_tstride : a.g_tstride;
                gx = __ldcg(reinterpret_cast<const float4*>(gp));
            }
        }
        uint32_t* const record0 = reinterpret_cast<uint32_t*>(a.set + (size_t)cta * stride + slot) + (gu >> 1);
        __half* yp = a.y + (size_t)(a.reverse ? T - 1 : 0) * a.y_tstride + (size_t)gn * a.y_bstride + u;   // output of the layer's next step
        const long y_step = a.reverse ? -a.y_tstride : a.y_tstride;
        const bool y_pairs = (reinterpret_cast<uintptr_t>(a.y) & 3) == 0 && a.y_tstride % 2 == 0 && a.y_bstride % 2 == 0;
        const float* const zp0 = zpart + layer * ZL + (gu * ZP + gn) * 4;
        for (int s = 0; s <= last; ++s) {
            uint32_t* const record = record0 + (unsigned)(s & 3) * (unsigned)buf * 4u;
            const float* zp = zp0 + (s & 1) * ZBUF;
            const int t_l = layer == 0 ? s : s - 2;              // the layer's step
            const bool act = live && t_l >= 0 && t_l < T;        // (a layer without a timestep repeats its state)
            float4 z = make_float4(gx.x + bias4.x, gx.y + bias4.y, gx.z + bias4.z, gx.w + bias4.w);
            asm volatile("bar.sync %0, %1;" ::"r"(1 + (s & 3)), "n"(kThreads) : "memory");   // the partial sums are there
            const bool lost = dead_step <= s;                    // or some are not (noted ahead of the barrier: the same for every gate thread)
            if (has_cells) {
                if (act) {
                    float4 q[kWarps];
#pragma unroll
                    for (int w = 0; w < kWarps; ++w) q[w] = *reinterpret_cast<const float4*>(zp + w * ZW);
#pragma unroll
                    for (int d = kWarps / 2; d > 0; d >>= 1)
#pragma unroll
                        for (int w = 0; w < d; ++w) { q[w].x += q[w + d].x; q[w].y += q[w + d].y; q[w].z += q[w + d].z; q[w].w += q[w + d].w; }
                    z.x += q[0].x; z.y += q[0].y; z.z += q[0].z; z.w += q[0].w;
                    c = sigmoidf_(z.y) * c + sigmoidf_(z.x) * tanhf_(z.z);
                    hh = __float2half_rn(sigmoidf_(z.w) * tanhf_(c));
                }
                if (lost) return;
                const uint32_t v = (uint32_t)__half_as_ushort(hh);
                const uint32_t pair = v | (__shfl_down_sync(0xffffffffu, v, 1, 8) << 16);
                if (live && s < last && (gu & 1) == 0) asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(record), "r"(pair) : "memory");
                if (act) {
                    if (layer == LAYERS - 1 && own) {
                        if (!y_pairs) *yp = hh;
                        else if ((gu & 1) == 0) *reinterpret_cast<uint32_t*>(yp) = pair;
                        yp += y_step;
                    }
                    if (layer == 0 && s + 1 < T) {               // next step's input-projection term
                        gp += g_step;
                        asm volatile("ld.global.cg.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(gx.x), "=f"(gx.y), "=f"(gx.z), "=f"(gx.w) : "l"(gp));
                    }
                }
            }
            if (lost) return;
            if (sweeps) {
                // sentinels for step s + 2; the fence ends ahead of the next barrier, and so of the records of step s + 1
                if (lane < padded) {
                    uint4* p = a.set + (size_t)((s + 2) & 3) * buf + (size_t)cta * stride + lane;
                    asm volatile("st.relaxed.gpu.global.v4.b32 [%0], {%1,%1,%1,%1};" ::"l"(p), "r"(~0u) : "memory");
                }
                __threadfence();
            }
        }
        if (own) {
            if (a.hn[layer]) a.hn[layer][(size_t)gn * H + u] = hh;
            if (a.cn[layer]) a.cn[layer][(size_t)gn * H + u] = __float2half_rn(c);
        }
        return;
    }

    // ================================ product warps ================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;" ::: "memory");
    // this warp's blocks warp, warp + 8, ...: the lane's octet of block i is 4 * block + t4
    uint4 wf[LAYERS][kMaxBlocks][2][2], hv[LAYERS][NT][kMaxBlocks];
#pragma unroll
    for (int i = 0; i < kMaxBlocks; ++i) {
        const int o = 4 * (warp + kWarps * i) + t4;
#pragma unroll
        for (int l = 0; l < LAYERS; ++l) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                wf[l][i][q >> 1][q & 1] = make_uint4(0u, 0u, 0u, 0u);
                if (o < n_cta) wf[l][i][q >> 1][q & 1] = __ldg(reinterpret_cast<const uint4*>(a.Whh[l] + (size_t)(u0 * 4 + q * 8 + g) * H + 8 * o));
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {                       // the initial hidden states
                const int n = j * 8 + g;
                uint4 x = make_uint4(0u, 0u, 0u, 0u);
                if (o < n_cta && n < B && a.h0[l]) {
                    const __half* p = a.h0[l] + (size_t)n * H + 8 * o;
                    __half v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = p[e];      // any alignment
                    x = *reinterpret_cast<const uint4*>(v);
                }
                hv[l][j][i] = x;
            }
        }
    }
    float accB[2][4];                                            // layer B's input product, made a step ahead
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) accB[m][e] = 0.f;
    // The lane's records of a step, all asked for together and without conditions: lanes of sequences or octets that do not
    // exist read the last one that does (their products meet no output: a column of its own, or weights of zero)
    uint4 hold[kMaxBlocks];
    const uint4* src[NT];
    unsigned off[kMaxBlocks];
#pragma unroll
    for (int j = 0; j < NT; ++j) src[j] = a.set + min(j * 8 + g, B - 1);
#pragma unroll
    for (int i = 0; i < kMaxBlocks; ++i) off[i] = (unsigned)(min(4 * (warp + kWarps * i) + t4, n_cta - 1) * stride);
    auto ask = [&](int step) {
        const unsigned at = (unsigned)(step & 3) * (unsigned)buf;
#pragma unroll
        for (int l = 0; l < LAYERS; ++l)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int i = 0; i < kMaxBlocks; ++i) hv[l][j][i] = ld_relaxed(src[j] + (at + off[i] + (unsigned)(l * B)));
    };

    // Cycles from a step's handover to the first look at the next one's records.  A look that comes too early costs another
    // trip of some 900 cycles, and the more records there are the more it delays them.  Measured optima at H = 1024 (us per
    // step without and with): 1 sequence 1.34 / 1.30, 8 1.52 / 1.39, 16 2.46 / 2.04, wavefront of 1 1.86 / 1.81, of 8 2.37 / 2.17.
    // With fewer CTAs (H = 320 to 640) only the optimum of more than 8 records lies elsewhere (1.3 to 1.5 thousand cycles).
    const unsigned look = slots > 8 ? (n_cta > 96 ? 1900u : 1400u) : (LAYERS == 2 ? 1350u : (slots > 4 ? 1100u : 1000u));
    for (int s = 0; s <= last; ++s) {
        float* zb = zpart + (s & 1) * ZBUF + warp * ZW;
        // ---- this step's hidden states (published in step s - 1)
        if (s > 0) {
            int polls = 0;
            while (true) {
                bool all = true;
#pragma unroll
                for (int l = 0; l < LAYERS; ++l)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int i = 0; i < kMaxBlocks; ++i) all = all && arrived(hv[l][j][i]);
                all = __all_sync(0xffffffffu, all);
                // counted at the first look too: records are often there by then, and a limit of one is no wait at all
                if (++polls >= a.poll_limit || ((polls & 1023) == 0 && status_aborted(a.status, a.gen))) {
                    // the gate warps leave behind this step's barrier; the other product warps then wait in vain, too
                    if (lane == 0) {
                        status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
                        atomicMin(&dead_step, s);
                    }
                    __syncwarp();
                    asm volatile("bar.arrive %0, %1;" ::"r"(1 + (s & 3)), "n"(kThreads) : "memory");
                    return;
                }
                if (all) break;
                ask(s - 1);
            }
        }
        if (LAYERS == 2)
#pragma unroll
            for (int i = 0; i < kMaxBlocks; ++i) hold[i] = hv[0][0][i];   // for the input product, when hv takes the next ones
        float acc[LAYERS][NT][2][4];
#pragma unroll
        for (int l = 0; l < LAYERS; ++l)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[l][j][m][e] = (LAYERS == 2 && l == 1) ? accB[m][e] : 0.f;
#pragma unroll
        for (int i = 0; i < kMaxBlocks; ++i)
            if (warp + kWarps * i < blocks)                      // warp-uniform
#pragma unroll
                for (int l = 0; l < LAYERS; ++l)
#pragma unroll
                    for (int j = 0; j < NT; ++j) multiply(acc[l][j], wf[l][i], hv[l][j][i]);
        // rows are gate rows (unit * 4 + gate): the four gates of a cell side by side
        if (warp < blocks) {
#pragma unroll
            for (int l = 0; l < LAYERS; ++l)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int r = m * 16 + g + (e >> 1) * 8, n = j * 8 + 2 * t4 + (e & 1);
                            zb[l * ZL + ((r >> 2) * ZP + n) * 4 + (r & 3)] = acc[l][j][m][e];
                        }
        }
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + (s & 3)), "n"(kThreads) : "memory");
        const unsigned handed_over = clock();
        if (LAYERS == 2) {
            // ---- layer B's input product of the next step: B's step s - 1 takes A's output of that step, published in
            //      step s - 1 and held in `hold`
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e) accB[m][e] = 0.f;
#pragma unroll
            for (int i = 0; i < kMaxBlocks; ++i) {
                const int b = warp + kWarps * i;
                if (b < blocks) {
                    uint4 w[2][2];
#pragma unroll
                    for (int q = 0; q < 4; ++q) w[q >> 1][q & 1] = wib[(b * 4 + q) * 32 + lane];
                    multiply(accB, w, hold[i]);
                }
            }
        }
        // the first look at the next step's records, timed to meet them in L2
        if (s < last) {
            while ((unsigned)clock() - handed_over < look) {}
            ask(s);
        }
    }
}

}  // namespace

size_t direct_smem(int H, int layers) {
    const int zp = layers == 2 ? 9 : 17;                         // the larger of NT = 1 and 2
    const size_t wib = layers == 2 ? (size_t)((H / 8 + 3) / 4) * 4 * 32 * 16 : 0;
    return (size_t)2 * kWarps * layers * 8 * zp * 16 + wib;
}

int launch_lstm_direct(const DirectArgs& a, int layers, cudaStream_t st) {
    const void* fn = layers == 2 ? (const void*)lstm_direct_kernel<2, 1>
                                 : (a.B <= 8 ? (const void*)lstm_direct_kernel<1, 1> : (const void*)lstm_direct_kernel<1, 2>);
    const size_t smem = direct_smem(a.H, layers);
    // (always what the largest layer needs: the limit belongs to the function, and another thread may be about to launch it)
    PIMB200_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)direct_smem(8 * kDirectMaxCtas, layers)));
    void* kargs[] = {const_cast<DirectArgs*>(&a)};
    PIMB200_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(a.H / 8), dim3(kThreads), kargs, smem, st));
    return PIMB200_OK;
}

}  // namespace pimb200
