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
