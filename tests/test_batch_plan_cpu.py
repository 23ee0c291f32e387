"""CPU: sizes of the batched persistent kernels (csrc/batch_plan.h, compiled by the host compiler)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pimaicompiler_b200", "csrc")

SOURCE = r"""
#include "batch_plan.h"
using namespace pimb200::tc;
extern "C" {
size_t smem_per_sm() { return kSmemPerSm; }
size_t smem_per_cta() { return kSmemPerCta; }
size_t lstm_smem(int H, int nj, int subs) { return lstm_batch_smem(H, nj, subs); }
void batch(int B, int most, int* out) {
    const LstmBatchPlan p = lstm_batch_plan(B, most);
    out[0] = p.groups, out[1] = p.subs, out[2] = p.nj;
}
int stages(int nj) { return stages_of(nj); }
int per_stage(int nj) { return blocks_per_stage(nj); }
void debt(unsigned q, unsigned leader, unsigned other, unsigned bytes, unsigned* out) {
    const StageDebt d = stage_debt(q, leader, other, bytes);
    out[0] = d.expect;
    out[1] = d.credit;
}
unsigned first_open(unsigned uses, unsigned stages) { return first_open_use(uses, stages); }
unsigned use_blocks(unsigned q, unsigned blocks, unsigned per_use) { return blocks_of_use(q, blocks, per_use); }
void greedy(int PH, int JH, size_t smem, int resident, int* out) {
    GreedyPlan p = greedy_plan(PH, JH, smem);
    p.groups = greedy_groups(p, resident);
    out[0] = p.ctas, out[1] = p.jrows, out[2] = p.groups, out[3] = p.max_nj, out[4] = p.capacity();
}
size_t greedy_smem(int PH, int JH, int utts) { return greedy_batch_smem(PH, joint_rows(JH, PH / 32), utts); }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-I", CSRC, "-o", d / "plan.so", d / "plan.cpp"], check=True)
    lib = ctypes.CDLL(str(d / "plan.so"))
    for f in (lib.smem_per_sm, lib.smem_per_cta, lib.lstm_smem, lib.greedy_smem):
        f.restype = ctypes.c_size_t
    return lib


def test_a_cta_of_the_batched_kernels_has_its_sm_for_itself(plan):
    # each takes all 512 columns of tensor memory: a second one on the SM would wait for them without a bound
    reserved = 1024                                    # of every CTA, by the system
    sizes = [plan.lstm_smem(H, nj, subs) for H in range(64, 1025, 64) for nj in (1, 2, 3, 4, 5, 6, 8) for subs in (1, 2)]
    sizes += [plan.greedy_smem(PH, JH, utts) for PH in range(64, 321, 64) for JH in (8, 64, 128, 512) if JH <= 2 * PH for utts in range(16, 81, 16)]
    for smem in sizes:
        assert 2 * (smem + reserved) > plan.smem_per_sm()
        assert smem <= plan.smem_per_cta()


def test_groups_of_the_greedy_loop_have_all_their_ctas_resident(plan):
    out = (ctypes.c_int * 5)()

    def of(PH, JH, resident, smem=227 * 1024):
        plan.greedy(PH, JH, ctypes.c_size_t(smem), resident, out)
        return tuple(out)

    assert of(320, 512, 148) == (10, 52, 14, 5, 1120)
    assert of(320, 512, 9)[4] == 0 and of(320, 512, 10)[2] == 1       # fewer than a group has: the clusters take the call
    for resident in (0, 1, 9, 74, 132, 148, 296):
        ctas, _, groups, max_nj, capacity = of(320, 512, resident)
        assert groups * ctas <= min(resident, 148) and capacity == groups * max_nj * 16
    assert of(320, 1000, 148)[4] == 0                                 # more joint rows per CTA than one K block
    assert of(320, 512, 148, smem=150 * 1024)[3] < 5 and of(320, 512, 148, smem=100 * 1024)[4] == 0


def test_every_batch_has_an_instance_of_the_recurrence(plan):
    instances = {(1, 1), (2, 1), (2, 2), (3, 2), (4, 2), (5, 2), (6, 2), (8, 2)}       # those that are compiled
    out, seen = (ctypes.c_int * 3)(), set()
    for most in (1, 2, 4, 7, 14, 37, 74):
        for B in range(1, 256 * most + 1):
            plan.batch(B, most, out)
            groups, subs, nj = out
            assert 1 <= groups <= most and groups * subs * nj * 16 >= B > (groups - 1) * subs * nj * 16
            seen.add((nj, subs))
    assert seen == instances


class _Barrier:
    """A barrier of one arrival per phase that also counts bytes: a phase ends when neither is outstanding."""

    def __init__(self):
        self.phase, self.arrivals, self.bytes = 0, 1, 0

    def add(self, arrivals=0, expect=0, landed=0):
        self.bytes += expect - landed
        self.arrivals -= arrivals
        assert self.arrivals >= 0
        if self.arrivals == 0 and self.bytes == 0:
            self.phase, self.arrivals = self.phase + 1, 1


@pytest.mark.parametrize("nj", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("blocks", [1, 3, 5, 16])
def test_a_pair_that_gave_up_waits_for_every_copy_of_both_ctas(plan, nj, blocks):
    # whichever CTA got further, and whichever copies had landed before: behind the leader's drain all have
    stages, per = plan.stages(nj), plan.per_stage(nj)
    block_bytes, steps = nj * 1024, 4
    sizes = [min(per, blocks - k) for _ in range(steps) for k in range(0, blocks, per)]
    assert [plan.use_blocks(q, blocks, per) for q in range(len(sizes))] == sizes
    debt = (ctypes.c_uint * 2)()
    for leader in range(len(sizes) + 1):
        for other in range(max(0, leader - stages), min(len(sizes), leader + stages) + 1):
            done = max(0, max(leader, other) - stages)        # uses that were multiplied: all their copies have landed
            if done > min(leader, other):
                continue
            for early in range(4):                            # copies of the open uses that land ahead of the drain: of whom
                bars = [_Barrier() for _ in range(stages)]
                late = []
                for q in range(max(leader, other)):
                    half, bar = sizes[q] * block_bytes, bars[q % stages]
                    if q < other and (q < done or early & 1):
                        bar.add(landed=half)                  # (may come before the leader expects it)
                    elif q < other:
                        late.append((q, half))
                    if q < leader:
                        bar.add(arrivals=1, expect=2 * half)
                        if q < done or early & 2:
                            bar.add(landed=half)
                        else:
                            late.append((q, half))
                for q in range(plan.first_open(max(leader, other), stages), max(leader, other)):
                    half = sizes[q] * block_bytes
                    plan.debt(q, leader, other, half, debt)
                    if debt[0]:
                        bars[q % stages].add(arrivals=1, expect=debt[0])
                    if debt[1]:
                        bars[q % stages].add(landed=debt[1])
                    mine = [h for u, h in late if u == q]
                    for h in mine:                            # not before the last one
                        assert bars[q % stages].phase == q // stages
                        bars[q % stages].add(landed=h)
                    assert bars[q % stages].phase == q // stages + 1 and bars[q % stages].bytes == 0
