// RNN-T greedy decoding of many utterances in lock step, one persistent launch for all frames.
//
// A group of PH / 32 CTAs (10 for 320 prediction units) holds the prediction network and the joint: a CTA the 128 gate rows of
// 32 units of all three recurrent matrices and a slice of the joint's hidden units.  Two of the matrices lie in tensor memory
// (as A operands), the rest in shared memory.  Every group walks its own utterances, up to 80 of them, as the N operand of
// tcgen05.mma.  With one label per frame all utterances are always at the same frame.  Per frame, for the whole group:
//
//   layer 0: gates(P0[label] + Whh0 h0), h0 to all CTAs      the product is ready before the label is known
//   layer 1: gates(Wih1 h0 + Whh1 h1), h1 to all CTAs        the second product too; Whh0 h0 runs under this exchange
//   joint:   z slice = relu(E + W1p h1), partial logits W2 z from the CTA's slice, to all CTAs
//   label:   every CTA adds the partial logits of its share of the utterances and sends the arg max to all CTAs
//
// What bounds it: four exchanges through L2 per frame (write, fence, counter, poll, TMA load), and the special-function unit
// in the gates.  The 8-utterance clusters of rnnt_greedy_mma_kernel exchange faster (through distributed shared memory), but
// seven of them take 56 utterances a round: 4.9 us per frame and round, 19 rounds for 1024 utterances.  A frame of all of them
// takes 16.7 us here, of 448 utterances 15, of 112..224 8.9..9.6.
//
// Buffers are written again only after an exchange that every CTA joins later: h0 of the next evaluation follows the
// partial logits, which every CTA sends after it has loaded h0 and h1; the partial logits of the next frame follow the labels.  Utterances without a label keep their states.
// Every wait of the loops is bounded; on giving up a CTA records the error, lets its copies land and frees its tensor memory.
// The allocation of tensor memory has no bound and finds it free: a CTA has its SM's shared memory for itself.
#include "rnnt_batch.cuh"

#include <algorithm>

#include "batch_plan.h"
#include "gemm_rows.cuh"
#include "pimb200_rnnt.h"
#include "tc_common.cuh"

namespace pimb200 {
namespace tc {
namespace {

constexpr int kThreads = 352;          // TMA, MMA, TMEM owner, eight epilogue warps
constexpr int kFirstEpi = 3;
constexpr int kEpiWarps = 8;
constexpr int kUnits = 32;
constexpr int kMaxBlocks = 5;          // PH <= 320: two matrices of 32 TMEM columns per K block of 64
constexpr int kMaxUtts = kGreedyMaxUtts;   // per group
static_assert(kGreedyMaxJointRows == 64, "a CTA's joint rows are one K block of the product with W2");
constexpr int kVocab = kGreedyVocab;
constexpr int kACol = 192;             // TMEM: accumulators of layer 0 and of everything else at 0 and 96, Whh0, Whh1 from here
constexpr int kCounterWords = 32;      // a counter has a 128-byte line
constexpr int kExchanges = 3;          // h0, h1, partial logits
constexpr int kMaxCtas = kGreedyMaxCtas;

struct GreedyMaps {
    CUtensorMap h[2];                  // [utterances of all groups][PH], boxes of 64 units x one group
};

__device__ __forceinline__ void count_up(uint32_t* p) { asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory"); }
__device__ __forceinline__ void mbar_arrive_one(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// 8 columns of 32 TMEM lanes: r[c] = column c of the thread's lane
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// Lane l < n waits for its counter to reach `target`; false = gave up.  The values behind the counters may be read afterwards.
__device__ __forceinline__ bool wait_counters(const uint32_t* counter, bool mine, uint32_t target, const GreedyBatchArgs& a) {
    bool ready = !mine;
    for (int polls = 1; !__all_sync(0xffffffffu, ready); ++polls) {
        const bool lost = polls >= a.poll_limit || ((polls & 255) == 0 && status_aborted(a.status, a.gen));
        if (__any_sync(0xffffffffu, lost)) return false;
        if (!ready) {
            uint32_t v;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if (v >= target) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
                ready = true;
            }
        }
    }
    __syncwarp();
    return true;
}

// NJ: utterances of a group / 16
template <int NJ>
__global__ void __launch_bounds__(kThreads, 1) rnnt_greedy_batch_kernel(const __grid_constant__ GreedyMaps maps, const __grid_constant__ GreedyBatchArgs a) {
    constexpr int UTTS = 16 * NJ, HALF = 8 * NJ;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int PH = a.PH, blocks = PH >> 6, C = a.ctas;
    const int jpad = (a.jrows + 7) / 8 * 8;
    const GreedySmem at = greedy_layout(PH, a.jrows, UTTS);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + at.bars);
    // h0 arrived [blocks], h1 arrived [blocks], then: layer-0 sums, layer-1 sums, joint sums, logits sums ready; layer-0 sums read,
    // layer-1 sums read, z written, partial logits read, labels known, seen by the TMA warp, labels
    // in shared memory, all products done
    const uint32_t in0 = smem_u32(bars), bar0 = in0 + 8 * 2 * kMaxBlocks;
    enum { kSum0, kSum1, kSumJ, kSumL, kRead0, kRead1, kZ, kReadL, kLabels, kSeen, kEpi, kDone, kBars };
    auto bar = [&](int i) { return bar0 + 8 * i; };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxBlocks + kBars);
    volatile int* emits = reinterpret_cast<volatile int*>(tmem_slot + 1);      // does any utterance of the frame emit? [frame parity]
    int* label = reinterpret_cast<int*>(tmem_slot + 4);                         // [kMaxUtts]
    int* n_emit = label + kMaxUtts;                                             // [kMaxUtts]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % C, grp = (int)blockIdx.x / C;
    const int u0 = rank * kUnits, j0 = rank * a.jrows, utt0 = grp * UTTS;
    const int jrows = max(0, min(a.jrows, a.JH - j0));
    const volatile int* abort_flag = a.status + 1;
    uint32_t* const counters = a.counters + (size_t)grp * C * kExchanges * kCounterWords;
    auto counter = [&](int x, int cta) { return counters + ((size_t)x * C + cta) * kCounterWords; };

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2 * kMaxBlocks; ++i) mbar_init(in0 + 8 * i, 1);
        for (int i = 0; i < kBars; ++i) mbar_init(bar(i), i == kRead0 || i == kRead1 || i == kZ || i == kReadL || i == kLabels || i == kEpi ? kEpiWarps : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // weights to shared memory: K-major tiles of 64 columns, 128-byte swizzle
    for (int i = threadIdx.x; i < blocks * 1024; i += kThreads) {
        const int kb = i >> 10, row = (i >> 3) & 127, chunk = i & 7;
        *reinterpret_cast<uint4*>(smem + at.wih1 + kb * 16384 + tile_offset(row, chunk)) =
            __ldg(reinterpret_cast<const uint4*>(a.Wih1 + (size_t)(u0 * 4 + packed_row(row)) * PH + kb * 64) + chunk);
    }
    for (int i = threadIdx.x; i < blocks * jpad * 8; i += kThreads) {
        const int kb = i / (jpad * 8), row = (i >> 3) % jpad, chunk = i & 7;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (row < jrows) v = __ldg(reinterpret_cast<const uint4*>(a.W1p + (size_t)(j0 + row) * PH + kb * 64) + chunk);
        *reinterpret_cast<uint4*>(smem + at.w1p + kb * jpad * 128 + tile_offset(row, chunk)) = v;
    }
    for (int i = threadIdx.x; i < kVocab * 64; i += kThreads) {        // W2[:, slice], zeros behind the slice and the vocabulary
        const int row = i >> 6, k = i & 63;
        __half v = __float2half_rn(0.f);
        if (row < a.V && k < jrows) v = a.W2[(size_t)row * a.JH + j0 + k];
        *reinterpret_cast<__half*>(smem + at.w2 + tile_offset(row, k >> 3) + (k & 7) * 2) = v;
    }
    for (int i = threadIdx.x; i < kMaxUtts; i += kThreads) {
        label[i] = a.blank;            // the start-of-sequence evaluation embeds the blank symbol
        n_emit[i] = 0;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    if (warp >= kFirstEpi && warp < kFirstEpi + 4) {
        const int q = warp & 3;
        for (int m = 0; m < 2; ++m) {
            const __half* src = (m ? a.Whh1 : a.Whh0) + (size_t)(u0 * 4 + packed_row(32 * q + lane)) * PH;
            for (int kb = 0; kb < blocks; ++kb) {
                uint32_t w[32];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + kb * 64) + i);
                    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
                }
                tmem_st32(tmem_base + ((uint32_t)(32 * q) << 16) + kACol + 32 * (m * blocks + kb), w);
            }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    bool failed = false;
    // the flow of a frame for every role: an evaluation of the prediction network if the frame before emitted anything
    // (frame 0: the start of sequence), then joint, logits and labels.  `evals` counts evaluations
    if (warp == 0) {
        // ---------------- TMA: states of the whole group ----------------
        const uint32_t el = elect_one();
        uint32_t evals = 0, loads[2] = {0, 0};
        for (int t = 0; t < a.Tp && !failed; ++t) {
            if (t > 0) {
                if (__any_sync(0xffffffffu, !mbar_wait(bar(kLabels), (uint32_t)((t - 1) & 1), abort_flag, a.gen))) { failed = true; break; }
                const bool eval = emits[(t - 1) & 1] != 0;
                __syncwarp();
                if (lane == 0) mbar_arrive_one(bar(kSeen));
                if (!eval) continue;
            }
            ++evals;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                if (!failed && !wait_counters(counter(x, lane < C ? lane : 0), lane < C, kEpiWarps * evals, a)) failed = true;
                if (failed) break;
                ++loads[x];
                for (int kb = 0; kb < blocks; ++kb) {
                    const uint32_t b = in0 + 8 * (x * kMaxBlocks + kb);
                    expect_tx_if(el, b, UTTS * 128);
                    load_2d<1>(el, smem_u32(smem + at.h[x] + kb * UTTS * 128), &maps.h[x], b, kb * 64, utt0);
                }
            }
        }
        if (failed && lane == 0) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
        // let the copies already issued land before the shared memory is given back
        if (lane == 0) {
#pragma unroll
            for (int x = 0; x < 2; ++x)
                for (int kb = 0; loads[x] > 0 && kb < blocks; ++kb)
                    for (uint32_t i = 0; i < (1u << 20); ++i)
                        if (mbar_try_wait(in0 + 8 * (x * kMaxBlocks + kb), (loads[x] - 1) & 1)) break;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t el = elect_one();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(UTTS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t d_wih1 = make_smem_desc(smem_u32(smem + at.wih1)), d_w1p = make_smem_desc(smem_u32(smem + at.w1p)),
                       d_w2 = make_smem_desc(smem_u32(smem + at.w2)), d_h0 = make_smem_desc(smem_u32(smem + at.h[0])),
                       d_h1 = make_smem_desc(smem_u32(smem + at.h[1]));
        const uint32_t acc0 = tmem_base, acc1 = tmem_base + 96, whh0 = tmem_base + kACol, whh1 = whh0 + 32 * blocks;
        uint32_t evals = 0;
        auto wait = [&](uint32_t b, uint32_t parity) {
            if (!failed && !mbar_wait(b, parity, abort_flag, a.gen)) failed = true;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return !failed;
        };
        for (int t = 0; t < a.Tp && !failed; ++t) {
            bool eval = t == 0;
            if (t > 0) {
                if (!wait(bar(kLabels), (uint32_t)((t - 1) & 1))) break;
                eval = emits[(t - 1) & 1] != 0;
            }
            if (eval) {
                const uint32_t par = evals & 1;
                // layer 1 (its state product is there already, but for the first evaluation)
                for (int kb = 0; kb < blocks; ++kb) {
                    if (!wait(in0 + 8 * kb, par)) break;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mma<1>(el, acc1, d_wih1 + (uint64_t)(kb * 1024 + 2 * k), d_h0 + (uint64_t)(kb * UTTS * 8 + 2 * k), idesc, evals > 0 || kb > 0 || k > 0 ? 1u : 0u);
                }
                if (failed) break;
                commit<1>(el, bar(kSum1));
                // layer 0 of the next evaluation
                if (!wait(bar(kRead0), par)) break;
                for (int kb = 0; kb < blocks; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mma_ta<1>(el, acc0, whh0 + 32 * kb + 8 * k, d_h0 + (uint64_t)(kb * UTTS * 8 + 2 * k), idesc, kb > 0 || k > 0 ? 1u : 0u);
                commit<1>(el, bar(kSum0));
                if (!wait(bar(kRead1), par)) break;
                for (int kb = 0; kb < blocks; ++kb)
                    if (!wait(in0 + 8 * (kMaxBlocks + kb), par)) break;
                if (failed) break;
                ++evals;
            }
            for (int kb = 0; kb < blocks; ++kb)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma<1>(el, acc1, d_w1p + (uint64_t)(kb * jpad * 8 + 2 * k), d_h1 + (uint64_t)(kb * UTTS * 8 + 2 * k), idesc, kb > 0 || k > 0 ? 1u : 0u);
            commit<1>(el, bar(kSumJ));
            if (!wait(bar(kZ), (uint32_t)(t & 1))) break;
#pragma unroll
            for (int k = 0; k < 4; ++k) mma<1>(el, acc1, d_w2 + (uint64_t)(2 * k), d_h0 + (uint64_t)(2 * k), idesc, k > 0 ? 1u : 0u);
            commit<1>(el, bar(kSumL));
            if (!wait(bar(kReadL), (uint32_t)(t & 1))) break;
            // the state product of the next layer 1
            for (int kb = 0; kb < blocks; ++kb)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma_ta<1>(el, acc1, whh1 + 32 * kb + 8 * k, d_h1 + (uint64_t)(kb * UTTS * 8 + 2 * k), idesc, kb > 0 || k > 0 ? 1u : 0u);
        }
        if (failed && lane == 0) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
        __syncwarp();
        commit<1>(el, bar(kDone));
        for (uint32_t i = 0; i < (1u << 20); ++i)      // no product is under way when the tensor memory is given back
            if (mbar_try_wait(bar(kDone), 0)) break;
    } else if (warp >= kFirstEpi) {
        // ---------------- gates, joint, labels ----------------
        const int ew = warp - kFirstEpi, q = warp & 3, hf = ew >> 2;
        const int r = lane >> 2, cq = lane & 3;
        const int unit = u0 + 8 * q + r, col = hf * HALF + 2 * cq;
        const uint32_t lanes = tmem_base + ((uint32_t)(32 * q) << 16);
        const float4 bias1 = __ldg(reinterpret_cast<const float4*>(a.bias1) + unit);
        const float b2 = lane < a.V ? a.b2[lane] : 0.f;
        float c0[NJ][2], c1[NJ][2];
#pragma unroll
        for (int j = 0; j < NJ; ++j) c0[j][0] = c0[j][1] = c1[j][0] = c1[j][1] = 0.f;
        const int valid = min(UTTS, a.n_utts - utt0);
        const int per = (UTTS + C - 1) / C;                            // utterances whose labels a CTA finds
        uint32_t* const words = a.labels + (size_t)grp * kMaxUtts;     // (frame + 1) << 8 | label
        uint32_t evals = 0;
        auto wait = [&](uint32_t b, uint32_t parity) {
            const bool ok = !failed && mbar_wait(b, parity, abort_flag, a.gen);
            if (__any_sync(0xffffffffu, !ok)) failed = true;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return !failed;
        };
        auto read_done = [&](int i) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_one(bar(i));
        };
        // E of the joint rows of this warp (lane quarters 0 and 1 hold them): into L2 a frame ahead, into registers while the
        // exchange ahead of the joint is under way
        float e[HALF];
        const int jr = 32 * q + lane;
        const bool joint_warp = q < 2, e_ok = joint_warp && jr < jrows;
        const float* const e_base = a.E + (long)(utt0 + hf * HALF) * a.e_utt + j0 + jr;
        auto load_e = [&](int t) {
            if (joint_warp) {
                const float* p = e_base + (long)t * a.e_frame;          // (a running address: forty products would be kept in registers)
#pragma unroll
                for (int i = 0; i < HALF; ++i, p += a.e_utt) e[i] = e_ok && hf * HALF + i < valid ? __ldcg(p) : 0.f;
            }
        };
        auto prefetch_e = [&](int t) {
            if (joint_warp && 32 * q < jrows)
                for (int i = lane; i < HALF && hf * HALF + i < valid; i += 32)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(e_base - lane + (long)i * a.e_utt + (long)t * a.e_frame));
        };
        // gates of this thread's cells: sums at `acc` (if there are any), input terms from `term`; the new h of the
        // utterances that `live` names to the exchange buffer
        auto cells = [&](uint32_t acc, bool has, float (&c)[NJ][2], auto&& term, __half* out, int read) {
            uint32_t hv[NJ];
            bool live[NJ][2];
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int2 tok = *reinterpret_cast<const int2*>(label + col + 8 * j);
                live[j][0] = evals == 0 || tok.x != a.blank;
                live[j][1] = evals == 0 || tok.y != a.blank;
            }
            // up to three column octets at a time: their cells' chains run side by side
#pragma unroll
            for (int j0 = 0; j0 < NJ; j0 += 3) {
                float4 x[3][2];
                uint32_t v[3][8];
#pragma unroll
                for (int j = j0; j < NJ && j < j0 + 3; ++j) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) x[j - j0][i] = term(j, i);
                    if (has) {
                        tmem_ld_16x256(acc + hf * HALF + 8 * j, v[j - j0]);
                        tmem_ld_16x256(acc + (16u << 16) + hf * HALF + 8 * j, v[j - j0] + 4);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[j - j0][i] = 0u;
                    }
                }
                if (has) tmem_wait_ld();
                if (j0 + 3 >= NJ) read_done(read);
#pragma unroll
                for (int j = j0; j < NJ && j < j0 + 3; ++j) {
                    float hj[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint32_t* z = v[j - j0] + i;
                        const float4 t = x[j - j0][i];
                        float cn = c[j][i];
                        hj[i] = lstm_cell(__uint_as_float(z[0]) + t.x, __uint_as_float(z[2]) + t.y, __uint_as_float(z[4]) + t.z, __uint_as_float(z[6]) + t.w, cn);
                        if (live[j][i]) c[j][i] = cn;
                    }
                    const __half2 hh = __floats2half2_rn(hj[0], hj[1]);
                    hv[j] = *reinterpret_cast<const uint32_t*>(&hh);
                }
            }
            // pairs of lanes swap: each has two units of one utterance
            const int b0 = r & 1;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, hv[j], 4);
                const uint32_t w = b0 ? __byte_perm(o, hv[j], 0x7632) : __byte_perm(hv[j], o, 0x5410);
                if (b0 ? live[j][1] : live[j][0]) *reinterpret_cast<uint32_t*>(out + (size_t)(utt0 + col + 8 * j + b0) * PH + u0 + 8 * q + 2 * (r >> 1)) = w;
            }
            asm volatile("fence.proxy.async.global;" ::: "memory");
            __syncwarp();
        };
        __half* const h0x = a.state;
        __half* const h1x = a.state + (size_t)(gridDim.x / C) * UTTS * PH;
        const size_t part_group = (size_t)C * UTTS * kVocab;
        for (int t = 0; t < a.Tp && !failed; ++t) {
            long long* tr = a.trace && blockIdx.x == 0 && threadIdx.x == kFirstEpi * 32 ? a.trace + (size_t)t * 8 : nullptr;
            if (tr) tr[0] = clock64();
            bool eval = t == 0;
            if (t > 0) eval = emits[(t - 1) & 1] != 0;
            if (eval) {
                const uint32_t par = evals & 1;
                if (evals > 0 && !wait(bar(kSum0), par ^ 1)) break;
                if (tr) tr[1] = clock64();
                cells(lanes, evals > 0, c0, [&](int j, int i) {
                    return __ldg(reinterpret_cast<const float4*>(a.P0 + (size_t)label[col + 8 * j + i] * 4 * PH) + unit);
                }, h0x, kRead0);
                if (lane == 0) count_up(counter(0, rank));
                if (tr) tr[2] = clock64();
                if (!wait(bar(kSum1), par)) break;
                if (tr) tr[3] = clock64();
                cells(lanes + 96, true, c1, [&](int, int) { return bias1; }, h1x, kRead1);
                if (lane == 0) count_up(counter(1, rank));
                if (tr) tr[4] = clock64();
                ++evals;
            }
            load_e(t);
            if (!wait(bar(kSumJ), (uint32_t)(t & 1))) break;
            if (tr) tr[5] = clock64();
            if (joint_warp) {
                // z = relu(E + Pj) of this lane's joint row for every utterance of the half, into the product's B tile; zeros
                // behind the slice (W2 is zero there, but what lies in the tile may be anything)
                unsigned char* const zt = smem + at.h[0];
#pragma unroll
                for (int i0 = 0; i0 < HALF; i0 += 8) {
                    uint32_t v[8];
                    tmem_ld8(lanes + 96 + hf * HALF + i0, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float p = __half2float(__float2half_rn(__uint_as_float(v[i])));
                        const float z = jr < jrows ? fmaxf(e[i0 + i] + p, 0.f) : 0.f;
                        *reinterpret_cast<__half*>(zt + tile_offset(hf * HALF + i0 + i, jr >> 3) + (jr & 7) * 2) = __float2half_rn(z);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            read_done(kZ);
            if (!wait(bar(kSumL), (uint32_t)(t & 1))) break;
            float* const part = a.partials + grp * part_group;
            if (q == 0) {
                uint32_t v[HALF];
#pragma unroll
                for (int i = 0; i < HALF; i += 8) tmem_ld8(lanes + 96 + hf * HALF + i, v + i);
                tmem_wait_ld();
                float* p = part + ((size_t)rank * UTTS + hf * HALF) * kVocab + lane;
#pragma unroll
                for (int i = 0; i < HALF; ++i) __stcg(p + i * kVocab, __uint_as_float(v[i]));
                __syncwarp();
                if (lane == 0) count_up(counter(2, rank));
            }
            read_done(kReadL);
            if (tr) tr[6] = clock64();
            if (t + 1 < a.Tp) prefetch_e(t + 1);
            // ---- labels: every CTA those of its own utterances, all partial logits in the same order; they go to the other CTAs
            //      as words that carry the frame, which the readers poll
            const int own0 = rank * per, own1 = min(UTTS, own0 + per);
            if (own0 + ew < own1) {
                if (!wait_counters(counter(2, lane < C ? lane : 0), lane < C, 2u * (uint32_t)(t + 1), a)) { failed = true; break; }
                if (tr) tr[7] = clock64();
                for (int n = own0 + ew; n < own1; n += kEpiWarps) {
                    const float* const mine = part + (size_t)n * kVocab + lane;
                    float sum = 0.f;
#pragma unroll 5
                    for (int k = 0; k < C; ++k) sum += __ldcg(mine + (size_t)k * UTTS * kVocab);
                    const float v = lane < a.V ? sum + b2 : -INFINITY;      // (0 x inf is a NaN)
                    // arg max over the 32 lanes, lowest index on ties, through an order-preserving integer image of the value
                    uint32_t key = __float_as_uint(v);
                    key = (key & 0x80000000u) ? ~key : (key | 0x80000000u);
                    const uint32_t kmax = __reduce_max_sync(0xffffffffu, key);
                    int best = min((int)__reduce_min_sync(0xffffffffu, key == kmax ? (uint32_t)lane : 0xffffffffu), a.V - 1);
                    if (n >= valid) best = a.blank;
                    if (lane == 0)
                        asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(words + n), "r"((uint32_t)(t + 1) << 8 | (uint32_t)best) : "memory");
                    if (n < valid) {
                        if (a.logits && lane < a.V) a.logits[((size_t)(utt0 + n) * a.Tp + t) * a.V + lane] = v;
                        if (lane == 0 && best != a.blank) {
                            a.tokens[(size_t)(utt0 + n) * a.Tp + n_emit[n]] = best;
                            ++n_emit[n];
                        }
                    }
                }
            }
            // every warp picks up an eighth of the labels
            {
                const int n = ew * (UTTS / kEpiWarps) + lane;
                bool here = lane >= UTTS / kEpiWarps;
                uint32_t w = 0;
                for (int polls = 1; !__all_sync(0xffffffffu, here); ++polls) {
                    const bool lost = polls >= a.poll_limit || ((polls & 255) == 0 && status_aborted(a.status, a.gen));
                    if (__any_sync(0xffffffffu, lost)) { failed = true; break; }
                    if (!here) {
                        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w) : "l"(words + n) : "memory");
                        here = w >> 8 == (uint32_t)(t + 1);
                    }
                }
                if (failed) break;
                if (lane < UTTS / kEpiWarps) label[n] = (int)(w & 0xffu);
            }
            // (no named barrier: a warp that gave up would never arrive, and no one else could leave)
            __syncwarp();
            if (lane == 0) mbar_arrive_one(bar(kEpi));
            if (!wait(bar(kEpi), (uint32_t)(t & 1))) break;
            bool any = false;
            for (int n = lane; n < UTTS; n += 32) any = any || label[n] != a.blank;
            any = __any_sync(0xffffffffu, any);
            if (t > 0 && !wait(bar(kSeen), (uint32_t)((t - 1) & 1))) break;      // (the TMA warp is never two frames behind)
            if (lane == 0) {
                emits[t & 1] = any;
                mbar_arrive_one(bar(kLabels));
            }
            __syncwarp();
        }
        if (failed) {
            if (lane == 0) status_raise(a.status, a.gen, PIMB200_ERR_TIMEOUT);
        } else {
            for (int n = rank * per + ew; n < min(valid, (rank + 1) * per); n += kEpiWarps)
                if (lane == 0) a.n_tokens[utt0 + n] = n_emit[n];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

using GreedyBatchFn = void (*)(GreedyMaps, GreedyBatchArgs);
GreedyBatchFn pick_nj(int nj) {
    switch (nj) {
        case 1: return rnnt_greedy_batch_kernel<1>;
        case 2: return rnnt_greedy_batch_kernel<2>;
        case 3: return rnnt_greedy_batch_kernel<3>;
        case 4: return rnnt_greedy_batch_kernel<4>;
        default: return rnnt_greedy_batch_kernel<5>;
    }
}

}  // namespace
}  // namespace tc

tc::GreedyPlan greedy_batch_plan(int PH, int JH, int V) {
    using namespace tc;
    GreedyPlan p = {};
    int dev = 0, sms = 0, smem = 0, per_sm = 0;
    if (PH <= 0 || PH % 64 != 0 || PH / 64 > kMaxBlocks || V > kVocab || cudaGetDevice(&dev) != cudaSuccess) return p;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    p = greedy_plan(PH, JH, (size_t)smem);
    if (p.max_nj == 0) return p;
    const GreedyBatchFn fn = pick_nj(p.max_nj);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerCta) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, greedy_batch_smem(PH, p.jrows, 16 * p.max_nj)) != cudaSuccess) {
        cudaGetLastError();
        return p;
    }
    p.groups = greedy_groups(p, sms * per_sm);
    return p;
}

void greedy_batch_workspace(int PH, size_t* state, size_t* partials, size_t* counters) {
    using namespace tc;
    const int ctas = PH / kUnits, groups = kMaxCtas / ctas;
    *state = (size_t)2 * groups * kMaxUtts * PH * 2;
    *partials = (size_t)groups * ctas * kMaxUtts * kVocab * 4;
    *counters = (size_t)groups * (ctas * kExchanges * kCounterWords + kMaxUtts) * 4;
}

int launch_greedy_batch(GreedyBatchArgs& a, const tc::GreedyPlan& p, cudaStream_t st) {
    using namespace tc;
    if (a.n_utts > p.capacity()) return PIMB200_ERR_UNSUPPORTED;
    int dev = 0, rc, gen;
    int* status;
    if ((rc = tc_prepare(&dev, &status, &gen)) != PIMB200_OK) return rc;     // (the tensor-map encoder)
    const int nj = ceil_div(ceil_div(a.n_utts, p.groups), 16), groups = ceil_div(a.n_utts, 16 * nj);
    a.ctas = p.ctas;
    a.jrows = p.jrows;
    GreedyMaps m = {};
    const size_t rows = (size_t)groups * 16 * nj;
    for (int x = 0; x < 2; ++x)
        if (!encode_2d(&m.h[x], a.state + x * rows * a.PH, rows, a.PH, (uint64_t)a.PH * 2, 16 * nj, 2)) return PIMB200_ERR_UNSUPPORTED;
    const GreedyBatchFn fn = pick_nj(nj);
    const int smem = (int)greedy_batch_smem(a.PH, a.jrows, 16 * nj);
    // (always the most that any launch asks for: the limit belongs to the function, and another thread may be about to launch it)
    PIMB200_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemPerCta));
    a.labels = a.counters + (size_t)groups * p.ctas * kExchanges * kCounterWords;
    PIMB200_CUDA_TRY(cudaMemsetAsync(a.counters, 0, (size_t)groups * (p.ctas * kExchanges * kCounterWords + kMaxUtts) * 4, st));
    void* args[] = {&m, &a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)fn, dim3(groups * p.ctas), dim3(kThreads), args, smem, st);
    if (e != cudaErrorCooperativeLaunchTooLarge) return cuda_status(e);
    cudaGetLastError();                        // (fewer CTAs resident than when the plan was made)
    return PIMB200_ERR_UNSUPPORTED;
}

}  // namespace pimb200
