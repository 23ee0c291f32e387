// Sizes of the batched persistent kernels (lstm_batch.cu, rnnt_batch.cu): plain C++, so that a host compiler takes it alone.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define PIMB200_HD __host__ __device__
#else
#define PIMB200_HD
#endif

namespace pimb200 {
namespace tc {

constexpr size_t kSmemPerSm = 228 * 1024, kSmemPerCta = 227 * 1024;
// Both kernels take all of an SM's tensor memory, so a second CTA on the SM would wait in its allocation, which has no bound,
// until the first is done; and the first may wait for the second's hidden states.  A small layer's CTA would leave room for it,
// so every launch asks for more than half of an SM's shared memory.
constexpr size_t kOneCtaPerSm = 116 * 1024;
PIMB200_HD constexpr size_t alone_on_sm(size_t smem) { return smem > kOneCtaPerSm ? smem : kOneCtaPerSm; }

// ---- recurrence of many sequences ----
constexpr int kBlockBytes = 128 * 128; // a K block (64 columns) of a CTA's weights
constexpr int kRingBytes = 96 * 1024;
constexpr int kMaxStages = 8;
// nj: eighths of the sequences of a CTA's half of a sub-batch; subs: sub-batches per group
PIMB200_HD constexpr int blocks_per_stage(int nj) { return nj > 4 ? 2 : 4; }
PIMB200_HD constexpr int stages_of(int nj) {
    return kRingBytes / (blocks_per_stage(nj) * nj * 1024) < kMaxStages ? kRingBytes / (blocks_per_stage(nj) * nj * 1024) : kMaxStages;
}
// TMEM: the accumulator of sub-batch b at column b * acc_cols, behind them as many K blocks of weights (32 columns each) as fit.
// An MMA of few columns is bound by its A operand: 74 cycles from shared memory, 37 from tensor memory, at up to 64 columns.
PIMB200_HD constexpr int acc_cols(int nj) { return (16 * nj + 31) / 32 * 32; }
PIMB200_HD constexpr int tmem_blocks(int nj, int subs) { return (512 - subs * acc_cols(nj)) / 32; }
inline size_t lstm_batch_smem(int H, int nj, int subs) {
    const int blocks = H / 64, t = tmem_blocks(nj, subs), own = blocks > t ? blocks - t : 0;
    return alone_on_sm((size_t)own * kBlockBytes + kRingBytes + 1024 /*align*/ + 512 /*barriers*/);
}

// Launch of B sequences where `most` groups are resident, each with up to 256: as many groups as there are, and two sub-batches where
// a group has more than the 32 columns that cost as much as 16
struct LstmBatchPlan {
    int groups, subs, nj;
};
inline LstmBatchPlan lstm_batch_plan(int B, int most) {
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    LstmBatchPlan p;
    p.groups = most < up(B, 16) ? most : up(B, 16);
    p.subs = up(B, p.groups) > 32 ? 2 : 1;
    p.nj = up(up(B, p.groups * p.subs), 16);
    if (p.nj == 7) p.nj = 8;               // (sixteen gate warps share an even number of octets)
    p.groups = up(B, p.subs * p.nj * 16);
    return p;
}

// Stage uses of a CTA pair, numbered from 0: each CTA asks for its half of use q's copies, and the bytes of both count at the
// leader's barrier of stage q % STAGES, where the leader expects them when it asks for its own half.  A pair that gave up may
// have asked for different numbers of uses.  What the leader then adds to the barrier of use q, so that its phase completes
// when every copy that was asked for has landed: bytes to expect (with the arrival), or bytes to count as landed that will
// never come.  (A use is asked for once the use STAGES before it was multiplied, so only the last STAGES can be incomplete.)
struct StageDebt {
    uint32_t expect, credit;
};
PIMB200_HD inline StageDebt stage_debt(uint32_t q, uint32_t leader_uses, uint32_t other_uses, uint32_t half_bytes) {
    return StageDebt{q >= leader_uses ? half_bytes : 0u, q >= other_uses ? half_bytes : 0u};
}
PIMB200_HD inline uint32_t first_open_use(uint32_t uses, uint32_t stages) { return uses > stages ? uses - stages : 0; }
// K blocks in use q: a sub-batch's step takes its `blocks` in uses of `per_use`
PIMB200_HD inline uint32_t blocks_of_use(uint32_t q, uint32_t blocks, uint32_t per_use) {
    const uint32_t k0 = q % ((blocks + per_use - 1) / per_use) * per_use;
    return blocks - k0 < per_use ? blocks - k0 : per_use;
}

// ---- greedy loop of many utterances ----
constexpr int kGreedyVocab = 32;
struct GreedySmem {                    // offsets behind the 1024-byte boundary
    int wih1, w1p, w2, h[2], bars, total;
};
PIMB200_HD inline int joint_rows(int JH, int ctas) { return ((JH + ctas - 1) / ctas + 3) / 4 * 4; }
PIMB200_HD inline GreedySmem greedy_layout(int PH, int jrows, int utts) {
    GreedySmem s;
    const int blocks = PH / 64, jpad = (jrows + 7) / 8 * 8;
    s.wih1 = 0;
    s.w1p = s.wih1 + blocks * 128 * 128;
    s.w2 = s.w1p + blocks * jpad * 128;
    s.h[0] = s.w2 + kGreedyVocab * 128;
    s.h[1] = s.h[0] + blocks * utts * 128;
    s.bars = s.h[1] + blocks * utts * 128;
    // an A operand has 128 rows: what lies behind the joint's and W2's is multiplied too, into lanes that nobody reads
    const int last = s.w1p + (blocks - 1) * jpad * 128, reach = (last > s.w2 ? last : s.w2) + 128 * 128;
    if (s.bars < reach) s.bars = reach;
    s.total = s.bars + 1024;
    return s;
}
constexpr int kGreedyMaxCtas = 148, kGreedyMaxUtts = 80, kGreedyMaxJointRows = 64;
struct GreedyPlan {                    // of a model; groups 0: not one of this size, or not on this device
    int ctas, jrows;                   // CTAs of a group, joint rows of each
    int groups, max_nj;                // groups of a launch, sixteenths of the utterances of a group
    int capacity() const { return groups * max_nj * 16; }
};
inline size_t greedy_batch_smem(int PH, int jrows, int utts) { return alone_on_sm((size_t)greedy_layout(PH, jrows, utts).total + 1024 /*align*/); }
// What fits a CTA's shared memory; then, as many groups as have all their CTAs resident at once
inline GreedyPlan greedy_plan(int PH, int JH, size_t smem) {
    GreedyPlan p = {};
    p.ctas = PH / 32;
    p.jrows = joint_rows(JH, p.ctas);
    if (p.jrows > kGreedyMaxJointRows) return p;
    while (p.max_nj < kGreedyMaxUtts / 16 && greedy_batch_smem(PH, p.jrows, 16 * (p.max_nj + 1)) <= smem) ++p.max_nj;
    return p;
}
inline int greedy_groups(const GreedyPlan& p, int resident_ctas) {
    return p.max_nj == 0 ? 0 : (resident_ctas < kGreedyMaxCtas ? resident_ctas : kGreedyMaxCtas) / p.ctas;
}

}  // namespace tc
}  // namespace pimb200
