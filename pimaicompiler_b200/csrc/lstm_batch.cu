// The recurrence of an LSTM layer over many lock-step sequences on the 5th-generation tensor cores.
//
//     Z[4H, b] = W_hh[4H, H] h[H, b]        c, h <- gates(G + bias + Z)        one persistent launch for all steps
//
// Weights stay on the chip for the whole launch.  A CTA pair (cta_group::2) owns 64 hidden units, each CTA the 128 gate rows of
// 32 of them as the M operand: 256 KB at H = 1024, half of them or more in tensor memory (an A operand may lie there), the others in
// shared memory.  H / 64 pairs hold the matrix, 16 at H = 1024, so 64 pairs make four groups that each walk their own sequences, up to
// 256, as two sub-batches: the products of one run under the gates and the exchange of the other.
//
// Hidden states are the N operand: a sub-batch's rows are fetched by TMA straight from the output tensor, each CTA of a pair
// half of them, so every state crosses from L2 to an SM once per pair.  Weight rows are ordered so that the four gates of a
// unit lie eight TMEM lanes apart: tcgen05.ld of 16 lanes x 256 bits then hands one thread all gates of its cells, and
// needs no exchange between threads.  Cell states stay in registers.
//
// Ordering between CTAs: a warp writes its cells' h, fences for the async proxy and counts up its pair's counter with a
// release; the TMA warps watch the counters (one lane each), acquire, and load K block k (the 64 units of pair k) as soon as
// pair k's sixteen warps have counted.  K blocks are multiplied in the same order whoever comes first.
// What bounds it: the chain of a step (states from L2, products, gates on the special-function unit, counters), of which two
// sub-batches hide a half.  A step at H = 1024 takes 5.5 us for 129 sequences, 6.3 for 512, 8.2 for 768 and 9.5 for 1024, where
// lstm_persistent_pipe_kernel takes 3.9 for every 128 (31 at 1024); the cycles of a step at 256..1024 sequences: states 1.1 k,
// products 3.3..6 k, commit 1.2 k, gates 2.6..5.4 k, counters 1.5..2.5 k.
//
// Sums of all K in one fp32 accumulator of tensor memory, where the kernels for fewer sequences add four quarters: the error of the
// outputs against 64 bits is the same to three digits (1024 units, 150..1000 sequences: 2.10e-4..2.30e-4, the rounding of the states).
//
// Every wait of the loops is bounded; on giving up a CTA records the error, lets its copies land and frees its tensor memory.
// What has no bound waits for no other CTA's progress: the allocation of tensor memory finds it free (a CTA has its SM's shared
// memory for itself), and both CTAs of a pair reach the barriers at either end.
#include "lstm_batch.cuh"

#include <algorithm>
#include <atomic>

#include "batch_plan.h"
#include "gemm_rows.cuh"
#include "tc_common.cuh"

namespace pimb200 {
namespace tc {
namespace {

constexpr int kFirstEpi = 3;            // warps: TMA, MMA, TMEM owner, then 8 or 16 for the gates
constexpr int kUnits = 32;             // hidden units per CTA
constexpr int kMaxBlocks = 16;         // H <= 1024

struct BatchMaps {
    CUtensorMap h[2], h0[2];           // boxes of 64 units x 8 NJ sequences
};

__device__ __forceinline__ float4 ldg_stream_f4(const float* p) {
    const uint4 v = ldg_stream_v4(p);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

// Gate warps: sixteen from 96 columns on (1024 sequences: a phase of 5.4 thousand cycles with eight), where a thread's share of
// the cells still fits its registers.
__host__ __device__ constexpr int gate_warps(int nj) { return nj >= 6 ? 16 : 8; }
__host__ __device__ constexpr int threads_of(int nj) { return (kFirstEpi + gate_warps(nj)) * 32; }

// NJ: eighths of the sequences of a CTA's half of a sub-batch (a sub-batch is 16 NJ columns); SUBS: sub-batches per group
template <int NJ, int SUBS>
__global__ void __launch_bounds__(threads_of(NJ), 1) lstm_batch_kernel(const __grid_constant__ BatchMaps maps, const __grid_constant__ BatchArgs a) {
    constexpr int KPS = blocks_per_stage(NJ), BLOCK = NJ * 1024, STAGE = KPS * BLOCK, STAGES = stages_of(NJ);
    constexpr int COLS = 16 * NJ, kThreads = threads_of(NJ), kEpiWarps = gate_warps(NJ);
    constexpr int PARTS = kEpiWarps / 4, OCT = 2 * NJ / PARTS;         // column parts of the gate warps, octets of columns per part
    static_assert(2 * NJ % PARTS == 0, "whole octets per warp");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int kTmemBlocks = tmem_blocks(NJ, SUBS), kACol = SUBS * acc_cols(NJ);
    const int blocks = a.H >> 6, tblocks = blocks < kTmemBlocks ? blocks : kTmemBlocks;
    unsigned char* ring = smem + (size_t)(blocks - tblocks) * kBlockBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kRingBytes);
    // full[STAGES], empty[STAGES], accumulator full[2], accumulator read[2], all products done; then the TMEM base and a count
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * STAGES, accf0 = empty0 + 8 * STAGES, acce0 = accf0 + 16, done0 = acce0 + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
    uint32_t* other_uses = tmem_slot + 1;         // of the leader: stage uses that the other CTA asked for
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)(blockIdx.x & 1), pair = (int)(blockIdx.x >> 1) % blocks, grp = (int)(blockIdx.x >> 1) / blocks;
    const int dir_groups = (int)(gridDim.x >> 1) / blocks / a.dirs, d = grp / dir_groups;
    const BatchDir& dir = a.dir[d];
    const int u0 = pair * 64 + rank * kUnits;                          // first hidden unit of this CTA
    const int seq0 = (grp - d * dir_groups) * SUBS * COLS;             // first sequence of this group
    const bool h_first = a.begin > 0 || dir.h0 != nullptr;             // the first step has a product
    const volatile int* abort_flag = a.status + 1;
    long long* const trace = blockIdx.x < (unsigned)a.trace_ctas ? a.trace : nullptr;
    auto step_time = [&](int s) { return dir.reverse ? a.T - 1 - (a.begin + s) : a.begin + s; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(accf0 + 8 * s, 1);
            mbar_init(acce0 + 8 * s, 2 * (kEpiWarps + (s == 0 ? 1 : 0)));
        }
        mbar_init(done0, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    const __half* W = dir.Whh + (size_t)u0 * 4 * a.H;
    for (int i = threadIdx.x; i < (blocks - tblocks) * 1024; i += kThreads) {
        const int kb = i >> 10, row = (i >> 3) & 127, chunk = i & 7;
        *reinterpret_cast<uint4*>(smem + (size_t)kb * kBlockBytes + tile_offset(row, chunk)) =
            __ldg(reinterpret_cast<const uint4*>(W + (size_t)packed_row(row) * a.H + (tblocks + kb) * 64) + chunk);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    if (warp >= kFirstEpi && warp < kFirstEpi + 4) {
        const int q = warp & 3;                                        // the lane quarter this warp may write
        const __half* src = W + (size_t)packed_row(32 * q + lane) * a.H;
        for (int kb = 0; kb < tblocks; ++kb) {
            uint32_t w[32];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + kb * 64) + i);
                w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
            }
            tmem_st32(tmem_base + ((uint32_t)(32 * q) << 16) + kACol + 32 * kb, w);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    pair_sync<2>();                               // barriers, weights and tensor memory of both CTAs are there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    bool failed = false;
    uint32_t asked = 0;                           // stage uses whose copies this CTA asked for (TMA warp)
    if (warp == 0) {
        // ---------------- TMA: this CTA's half of every sub-batch's rows ----------------
        const uint32_t el = elect_one();
        const uint32_t ring0 = smem_u32(ring), lead0 = mapa(full0, 0);
        uint32_t st = 0, par = 1;
        for (int s = 0; s < a.steps && !failed; ++s) {
            if (s == 0 && !h_first) continue;
            const int tp = step_time(s - 1);                           // the step before
#pragma unroll 1
            for (int b = 0; b < SUBS && !failed; ++b) {
                const int row = seq0 + b * COLS + rank * (COLS / 2);
                const bool from_h0 = a.begin + s == 0;
                const CUtensorMap* map = from_h0 ? &maps.h0[d] : &maps.h[d];
                const int fold = from_h0 ? 0 : tp % a.y_fold, tc = from_h0 ? 0 : tp / a.y_fold;
                const uint32_t* counter = a.counters + ((size_t)(grp * SUBS + b) * blocks + lane) * kBatchFlagWords;
                bool ready = s == 0 || lane >= blocks;
                for (int k0 = 0; k0 < blocks; k0 += KPS) {
                    const int k1 = k0 + KPS < blocks ? k0 + KPS : blocks;
                    const uint32_t need = (uint32_t)((1ull << k1) - (1ull << k0));
                    for (int polls = 1; (__ballot_sync(0xffffffffu, ready) & need) != need; ++polls) {
                        const bool lost = polls >= a.poll_limit || ((polls & 255) == 0 && *abort_flag == a.gen);
                        if (__any_sync(0xffffffffu, lost)) { failed = true; break; }
                        if (!ready) {
                            uint32_t v;
                            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                            if (v >= (uint32_t)(2 * kEpiWarps * s)) {
                                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                                ready = true;
                            }
                        }
                        __syncwarp();
                    }
                    if (failed) break;
                    if (trace && lane == 0 && b == 0 && k0 == 0) trace[((size_t)blockIdx.x * a.steps + s) * 8] = clock64();
                    if (trace && lane == 0 && b == 0 && k1 == blocks) trace[((size_t)blockIdx.x * a.steps + s) * 8 + 1] = clock64();
                    if (__any_sync(0xffffffffu, !mbar_wait(empty0 + 8 * st, par, abort_flag, a.gen))) { failed = true; break; }
                    if (rank == 0) expect_tx_if(el, full0 + 8 * st, 2u * (uint32_t)((k1 - k0) * BLOCK));
                    for (int k = k0; k < k1; ++k)
                        load_3d<2>(el, ring0 + st * STAGE + (k - k0) * BLOCK, map, lead0 + 8 * st, fold * a.H + k * 64, row, tc);
                    ++asked;
                    if (++st == STAGES) { st = 0; par ^= 1; }
                }
            }
        }
        if (lane == 0) {
            if (failed) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
            if (rank == 1) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(mapa(smem_u32(other_uses), 0)), "r"(asked) : "memory");
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the pair's leader) ----------------
        if (rank == 0) {
            const uint32_t el = elect_one();
            const uint32_t idesc = (1u << 4) | ((uint32_t)(COLS >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            const uint64_t wdesc = make_smem_desc(smem_u32(smem)), rdesc = make_smem_desc(smem_u32(ring));
            uint32_t st = 0, par = 0, uses = 0;
            for (int s = 0; s < a.steps && !failed; ++s) {
                if (s == 0 && !h_first) continue;
#pragma unroll 1
                for (int b = 0; b < SUBS && !failed; ++b) {
                    if (!mbar_wait(acce0 + 8 * b, (uses & 1) ^ 1, abort_flag, a.gen)) { failed = true; break; }
                    const uint32_t acc = tmem_base + acc_cols(NJ) * b;
                    for (int k0 = 0; k0 < blocks; k0 += KPS) {
                        if (!mbar_wait(full0 + 8 * st, par, abort_flag, a.gen)) { failed = true; break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (trace && lane == 0 && b == 0 && k0 == 0) trace[((size_t)blockIdx.x * a.steps + s) * 8 + 6] = clock64();
                        if (trace && lane == 0 && b == 0 && k0 + KPS >= blocks) trace[((size_t)blockIdx.x * a.steps + s) * 8 + 7] = clock64();
#pragma unroll
                        for (int i = 0; i < KPS; ++i) {
                            const int kb = k0 + i;
                            if (kb >= blocks) break;
                            const uint64_t bdesc = rdesc + (uint64_t)((st * STAGE + i * BLOCK) >> 4);
                            if (kb < tblocks) {
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    mma_ta<2>(el, acc, tmem_base + kACol + 32 * kb + 8 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                            } else {
                                const uint64_t adesc = wdesc + (uint64_t)((kb - tblocks) * (kBlockBytes >> 4));
#pragma unroll
                                for (int k = 0; k < 4; ++k) mma<2>(el, acc, adesc + 2 * k, bdesc + 2 * k, idesc, 1u);
                            }
                        }
                        commit<2>(el, empty0 + 8 * st);
                        if (++st == STAGES) { st = 0; par ^= 1; }
                    }
                    if (!failed) commit<2>(el, accf0 + 8 * b);
                }
                ++uses;
            }
            if (failed && lane == 0) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
            __syncwarp();
            commit<2>(el, done0);
        }
        // no product is under way when the tensor memory is given back
        if (!mbar_wait(done0, 0, abort_flag, a.gen))
            for (uint32_t i = 0; i < (1u << 20); ++i)
                if (mbar_try_wait(done0, 0)) break;
    } else if (warp == 2) {
        // ---------------- input terms of this CTA's units into L2, two steps ahead: 64 KB per sub-batch and CTA, wanted by all CTAs
        //                  at once, take longer from HBM than the phase they are asked for in ----------------
        const long g_step = dir.reverse ? -a.g_tstride : a.g_tstride;
        const float* g = dir.G + (dir.reverse ? (long)(a.steps - 1) * a.g_tstride : 0) + 4 * u0 + (lane & 3) * 32;   // four lines per sequence
        const int n = min(SUBS * COLS, a.B - seq0);
        uint32_t par = 0;
        for (int s = 0; s < a.steps; ++s) {
            for (int ahead = s == 0 ? 1 : 2; ahead <= 2; ++ahead)
                if (s + ahead < a.steps)
                    for (int i = lane >> 2; i < n; i += 8)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(g + ahead * g_step + (long)(seq0 + i) * a.g_bstride));
            g += g_step;
            if (s == 0 && !h_first) continue;
            if (__any_sync(0xffffffffu, !mbar_wait(accf0, par, abort_flag, a.gen))) break;
            par ^= 1;
            // (never two steps behind: the next products wait for this)
            if (lane == 0) asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(acce0, 0)) : "memory");
        }
    } else if (warp >= kFirstEpi) {
        // ---------------- gates: TMEM lane quarter = warp % 4, a part of the columns ----------------
        const int q = warp & 3, part = (warp - kFirstEpi) >> 2;
        const int r = lane >> 2, cq = lane & 3;
        const int unit = u0 + 8 * q + r;
        const int col = part * (COLS / PARTS) + 2 * cq;                      // this thread's first column; the others 8 j + {0, 1} on
        const float4 bias = __ldg(reinterpret_cast<const float4*>(dir.bias) + unit);
        float c[SUBS][OCT][2];
        const float* gp[SUBS];
        int left[SUBS];                                                // sequences from the thread's first column to the end
        const int t_low = dir.reverse ? a.steps - 1 : 0;
        const long g_step = dir.reverse ? -a.g_tstride : a.g_tstride;
#pragma unroll
        for (int b = 0; b < SUBS; ++b) {
            const int seq = seq0 + b * COLS + col;
            left[b] = a.B - seq;
            gp[b] = dir.G + (long)t_low * a.g_tstride + (long)seq * a.g_bstride + 4 * unit;
#pragma unroll
            for (int j = 0; j < OCT; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    c[b][j][e] = 0.f;
                    if (8 * j + e < left[b]) {
                        const size_t at = (size_t)(seq + 8 * j + e) * a.H + unit;
                        if (a.begin > 0) c[b][j][e] = a.c_state[d][at];
                        else if (dir.c0) c[b][j][e] = __half2float(dir.c0[at]);
                    }
                }
        }
        // input terms of the coming phase (a sub-batch's step), asked for behind the phase before
        float4 g[OCT][2];
#pragma unroll
        for (int j = 0; j < OCT; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                g[j][e] = 8 * j + e < left[0] ? ldg_stream_f4(gp[0] + (long)(8 * j + e) * a.g_bstride) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t par = 0;
        const int b0 = r & 1, b1 = r >> 1 & 1, b2 = r >> 2;
        for (int s = 0; s < a.steps && !failed; ++s) {
            const bool has = s > 0 || h_first, last = s + 1 == a.steps;
            const int t = step_time(s);
            __half* const yt = dir.y + (long)(t / a.y_fold) * a.y_tstride + (long)(t % a.y_fold) * a.H;
#pragma unroll
            for (int b = 0; b < SUBS; ++b) {
                if (failed) break;
                if (has) {
                    if (!mbar_wait(accf0 + 8 * b, par, abort_flag, a.gen)) {
                        status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
                        failed = true;
                    }
                    if (__any_sync(0xffffffffu, failed)) { failed = true; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                if (trace && lane == 0 && warp == kFirstEpi) trace[((size_t)blockIdx.x * a.steps + s) * 8 + 2 + 2 * b] = clock64();
                const uint32_t acc = tmem_base + ((uint32_t)(32 * q) << 16) + acc_cols(NJ) * b + part * (COLS / PARTS);
                const int nb = b + 1 < SUBS ? b + 1 : 0;
                const float* const gn = b + 1 < SUBS ? gp[nb] : gp[0] + g_step;
                const int n_left = b + 1 < SUBS || !last ? left[nb] : 0;
                uint32_t hv[OCT];
                // four column octets at a time: their cells' chains run side by side
#pragma unroll
                for (int j0 = 0; j0 < OCT; j0 += 4) {
                    uint32_t v[4][8];
                    if (has) {
#pragma unroll
                        for (int j = j0; j < OCT && j < j0 + 4; ++j) {
                            tmem_ld_16x256(acc + 8 * j, v[j - j0]);
                            tmem_ld_16x256(acc + (16u << 16) + 8 * j, v[j - j0] + 4);
                        }
                        tmem_wait_ld();
                        if (j0 + 4 >= OCT) {        // the accumulator may be written again
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(acce0 + 8 * b, 0)) : "memory");
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i >> 3][i & 7] = 0u;
                    }
#pragma unroll
                    for (int j = j0; j < OCT && j < j0 + 4; ++j) {
                        float hj[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float4 gx = g[j][e];
                            const uint32_t* z = v[j - j0] + e;
                            // input term + bias first, then the product
                            hj[e] = lstm_cell((gx.x + bias.x) + __uint_as_float(z[0]), (gx.y + bias.y) + __uint_as_float(z[2]),
                                              (gx.z + bias.z) + __uint_as_float(z[4]), (gx.w + bias.w) + __uint_as_float(z[6]), c[b][j][e]);
                        }
                        const __half2 hh = __floats2half2_rn(hj[0], hj[1]);
                        hv[j] = *reinterpret_cast<const uint32_t*>(&hh);
                    }
                }
                // eight lanes hold the eight units of an octet for the same two sequences per j: pairs of lanes swap, so that
                // each has two units of one sequence, then four units, then all eight of one sequence per four j
                uint32_t w[OCT];
#pragma unroll
                for (int j = 0; j < OCT; ++j) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, hv[j], 4);
                    w[j] = b0 ? __byte_perm(o, hv[j], 0x7632) : __byte_perm(hv[j], o, 0x5410);
                }
                const int seq = seq0 + b * COLS + col + b0;
                auto put = [&](__half* base, long pitch) {
                    if constexpr (OCT % 2 != 0) {
#pragma unroll
                        for (int j = 0; j < OCT; ++j)
                            if (seq + 8 * j < a.B)
                                *reinterpret_cast<uint32_t*>(base + (long)(seq + 8 * j) * pitch + u0 + 8 * q + 2 * (r >> 1)) = w[j];
                    } else {
                        uint2 x[OCT / 2 > 0 ? OCT / 2 : 1];
#pragma unroll
                        for (int m = 0; m < OCT / 2; ++m) {
                            const uint32_t o = __shfl_xor_sync(0xffffffffu, b1 ? w[2 * m] : w[2 * m + 1], 8);
                            x[m] = b1 ? make_uint2(o, w[2 * m + 1]) : make_uint2(w[2 * m], o);
                        }
                        if constexpr (OCT % 4 != 0) {
#pragma unroll
                            for (int m = 0; m < OCT / 2; ++m) {
                                const int n = seq + 8 * (2 * m + b1);
                                if (n < a.B) *reinterpret_cast<uint2*>(base + (long)n * pitch + u0 + 8 * q + 4 * b2) = x[m];
                            }
                        } else {
#pragma unroll
                            for (int m = 0; m < OCT / 4; ++m) {
                                const uint2 keep = b2 ? x[2 * m + 1] : x[2 * m], give = b2 ? x[2 * m] : x[2 * m + 1];
                                const uint32_t ox = __shfl_xor_sync(0xffffffffu, give.x, 16), oy = __shfl_xor_sync(0xffffffffu, give.y, 16);
                                const int n = seq + 8 * (4 * m + 2 * b2 + b1);
                                if (n < a.B)
                                    *reinterpret_cast<uint4*>(base + (long)n * pitch + u0 + 8 * q) =
                                        b2 ? make_uint4(ox, oy, keep.x, keep.y) : make_uint4(keep.x, keep.y, ox, oy);
                            }
                        }
                    }
                };
                put(yt, a.y_bstride);
                if (!last) {
                    asm volatile("fence.proxy.async.global;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counters + ((size_t)(grp * SUBS + b) * blocks + pair) * kBatchFlagWords) : "memory");
                    __syncwarp();
                } else {
                    if (a.begin + a.steps == a.T && dir.hn) put(dir.hn, a.H);
#pragma unroll
                    for (int j = 0; j < OCT; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (8 * j + e >= left[b]) continue;
                            const size_t at = (size_t)(seq0 + b * COLS + col + 8 * j + e) * a.H + unit;
                            if (a.begin + a.steps < a.T) a.c_state[d][at] = c[b][j][e];
                            else if (dir.cn) dir.cn[at] = __float2half_rn(c[b][j][e]);
                        }
                }
                if (trace && lane == 0 && warp == kFirstEpi) trace[((size_t)blockIdx.x * a.steps + s) * 8 + 3 + 2 * b] = clock64();
                // the next phase's input terms: behind the fence, which would wait for them (they come from HBM)
                const float* gq = gn;          // (a running address: the products of all cells would be kept in registers)
#pragma unroll
                for (int j = 0; j < OCT; ++j, gq += 8 * a.g_bstride) {
                    if (8 * j < n_left) g[j][0] = ldg_stream_f4(gq);
                    if (8 * j + 1 < n_left) g[j][1] = ldg_stream_f4(gq + a.g_bstride);
                }
            }
#pragma unroll
            for (int b = 0; b < SUBS; ++b) gp[b] += g_step;
            if (has) par ^= 1;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    pair_sync<2>();                               // nobody multiplies or asks for copies any more
    if (warp == 0 && rank == 0 && lane == 0) {
        // let every copy of both CTAs land, whoever gave up and where (all have, if nobody did)
        const uint32_t theirs = *other_uses, all = asked > theirs ? asked : theirs;
        for (uint32_t q = first_open_use(all, STAGES); q < all; ++q) {
            const uint32_t bar = full0 + 8 * (q % STAGES);
            const StageDebt debt = stage_debt(q, asked, theirs, blocks_of_use(q, blocks, KPS) * BLOCK);
            if (debt.expect) mbar_expect_tx(bar, debt.expect);
            if (debt.credit) mbar_complete_tx(bar, debt.credit);
            for (uint32_t i = 0; i < (1u << 20); ++i)
                if (mbar_try_wait(bar, (q / STAGES) & 1)) break;
        }
    }
    __syncwarp();
    pair_sync<2>();                               // neither CTA leaves while copies of the other may still signal it
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

using BatchFn = void (*)(BatchMaps, BatchArgs);
// one sub-batch has up to 32 columns, each of two more than 16
BatchFn pick(int nj, int subs) {
    if (subs == 1) return nj == 1 ? lstm_batch_kernel<1, 1> : lstm_batch_kernel<2, 1>;
    switch (nj) {
        case 2: return lstm_batch_kernel<2, 2>;
        case 3: return lstm_batch_kernel<3, 2>;
        case 4: return lstm_batch_kernel<4, 2>;
        case 5: return lstm_batch_kernel<5, 2>;
        case 6: return lstm_batch_kernel<6, 2>;
        default: return lstm_batch_kernel<8, 2>;
    }
}

void launch_config(cudaLaunchConfig_t& lc, cudaLaunchAttribute* at, int H, int nj, int subs, int ctas, cudaStream_t st) {
    lc = {};
    lc.gridDim = dim3(ctas);
    lc.blockDim = dim3(threads_of(nj));
    lc.dynamicSmemBytes = lstm_batch_smem(H, nj, subs);
    lc.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    lc.attrs = at;
    lc.numAttrs = 2;
}

// The most shared memory that any launch asks for, at every launch: the limit belongs to the function, and a thread with a handle of
// another size may be about to launch it
int raise_smem_limit(BatchFn fn) {
    return cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerCta));
}

// pairs of CTAs that are resident at once
int resident_pairs(int dev) {
    constexpr int kMaxDevices = 64;
    static std::atomic<int> pairs[kMaxDevices];     // (two threads that come first find the same)
    if (dev < 0 || dev >= kMaxDevices) return 0;
    int n = pairs[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchConfig_t lc;
        cudaLaunchAttribute at[2];
        launch_config(lc, at, 1024, 8, 2, 2, nullptr);
        lc.numAttrs = 1;
        if (raise_smem_limit(lstm_batch_kernel<8, 2>) != PIMB200_OK || cudaOccupancyMaxActiveClusters(&n, lstm_batch_kernel<8, 2>, &lc) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        n = n > 0 ? std::min(n, kBatchMaxPairs) : -1;
        pairs[dev].store(n, std::memory_order_relaxed);
    }
    return std::max(n, 0);
}

int groups_per_dir(int H, int dirs, int dev) {
    if (H % 64 != 0 || H <= 0 || H > 64 * kMaxBlocks) return 0;
    return resident_pairs(dev) / (H / 64) / dirs;
}

}  // namespace
}  // namespace tc

int lstm_batch_capacity(int H, int dirs) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    return tc::groups_per_dir(H, dirs, dev) * 256;
}

int launch_lstm_batch(BatchArgs& a, cudaStream_t st) {
    using namespace tc;
    int dev = 0, rc, gen;
    int* status;
    if ((rc = tc_prepare(&dev, &status, &gen)) != PIMB200_OK) return rc;
    const int most = groups_per_dir(a.H, a.dirs, dev);
    if (most == 0 || a.B > most * 256 || a.y_bstride % 8 != 0 || a.y_tstride % 8 != 0 || a.T % a.y_fold != 0) return PIMB200_ERR_UNSUPPORTED;
    for (int d = 0; d < a.dirs; ++d) {
        const BatchDir& r = a.dir[d];
        if (!aligned16(r.y) || (r.hn && !aligned16(r.hn)) || (r.h0 && !aligned16(r.h0)) || !aligned16(r.Whh)) return PIMB200_ERR_UNSUPPORTED;
    }
    const LstmBatchPlan plan = lstm_batch_plan(a.B, most);
    const int groups = plan.groups, subs = plan.subs, nj = plan.nj;
    BatchMaps m = {};
    for (int d = 0; d < a.dirs; ++d) {
        const BatchDir& r = a.dir[d];
        if (!encode_3d(&m.h[d], r.y, (uint64_t)a.H * a.y_fold, a.B, a.T / a.y_fold, (uint64_t)a.y_bstride * 2, (uint64_t)a.y_tstride * 2, 8 * nj)) return PIMB200_ERR_UNSUPPORTED;
        m.h0[d] = m.h[d];
        if (r.h0 && !encode_3d(&m.h0[d], r.h0, a.H, a.B, 1, (uint64_t)a.H * 2, (uint64_t)a.B * a.H * 2, 8 * nj)) return PIMB200_ERR_UNSUPPORTED;
    }
    const BatchFn fn = pick(nj, subs);
    const int blocks = a.H / 64;
    if ((rc = raise_smem_limit(fn)) != PIMB200_OK) return rc;
    PIMB200_CUDA_TRY(cudaMemsetAsync(a.counters, 0, (size_t)groups * a.dirs * subs * blocks * kBatchFlagWords * 4, st));
    cudaLaunchConfig_t lc;
    cudaLaunchAttribute at[2];
    launch_config(lc, at, a.H, nj, subs, 2 * groups * a.dirs * blocks, st);
    return cuda_status(cudaLaunchKernelEx(&lc, fn, m, a));
}

}  // namespace pimb200
