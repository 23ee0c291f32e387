"""GPU parity of the fused LSTM through the C ABI: both recurrence variants against the C oracle,
the libtorch golden fixtures, and libtorch CPU at the baseline's C1 shape."""
import glob
import os

import numpy as np
import pytest
import torch

from oracle import c_oracle as co
from tests.util import CONTRACT_ATOL, CONTRACT_RTOL, assert_close, device_memory_left, h16, lstm_params, to_dev

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")

# vs the fp32 oracle: h is rounded to fp16 every step (rel 2^-11 of values in (-1,1)) and the
# rounding feeds back through the recurrence; the contract bound is 2e-2 / 1e-2
LSTM_ATOL = 4e-3
LSTM_RTOL = 4e-3


def _ops():
    from pimaicompiler_b200 import ops
    return ops


def _run(ops, ps, x, h0, c0, L, bi, hb, bf, variant, bulk_wide=None):
    T = x.shape[1] if bf else x.shape[0]
    I, H = x.shape[2], ps[1].shape[1]
    m = ops.Lstm([to_dev(p) for p in ps], L, bi, I, H, hb)
    m.set_variant(variant)
    if bulk_wide is not None:   # None = the library's default choice of persistent kernel by batch size
        from pimaicompiler_b200 import _lib
        assert _lib.lib().pimb200_lstm_set_bulk_wide(m._h, bulk_wide) == 0
    y, hn, cn = m.forward(to_dev(x), None if h0 is None else to_dev(h0), None if c0 is None else to_dev(c0), bf)
    torch.cuda.synchronize()
    assert m.last_status() == 0
    return y, hn, cn


@pytest.mark.parametrize("path", sorted(p for p in glob.glob(os.path.join(GOLD, "lstm_*.npz")) if "packed" not in p))
def test_lstm_golden_streamed(path):
    ops = _ops()
    z = np.load(path)
    T, B, I, H, L, bi, hb, bf = [int(v) for v in z["cfg"]]
    ps, i = [], 0
    while f"p{i}" in z:
        ps.append(torch.from_numpy(z[f"p{i}"]).float())
        i += 1
    y, hn, cn = _run(ops, ps, torch.from_numpy(z["x"]).float(), torch.from_numpy(z["h0"]).float(),
                     torch.from_numpy(z["c0"]).float(), L, bool(bi), bool(hb), bool(bf), ops.LSTM_STREAMED)
    assert_close(y, z["y"], LSTM_ATOL, LSTM_RTOL, "y")
    assert_close(hn, z["hn"], LSTM_ATOL, LSTM_RTOL, "hn")
    assert_close(cn, z["cn"], LSTM_ATOL, LSTM_RTOL, "cn")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(GOLD, "lstm_packed_*.npz"))))
def test_lstm_golden_packed(path):
    ops = _ops()
    z = np.load(path)
    T, B, I, H, L, bi, hb, bf = [int(v) for v in z["cfg"]]
    ps, i = [], 0
    while f"p{i}" in z:
        ps.append(torch.from_numpy(z[f"p{i}"]).cuda())
        i += 1
    m = ops.Lstm(ps, L, bool(bi), I, H, True)
    y, hn, cn = m.forward_packed(torch.from_numpy(z["data"]).cuda(), torch.from_numpy(z["batch_sizes"]),
                                 torch.from_numpy(z["h0"]).cuda(), torch.from_numpy(z["c0"]).cuda())
    assert_close(y, z["y"], LSTM_ATOL, LSTM_RTOL, "packed y")
    assert_close(hn, z["hn"], LSTM_ATOL, LSTM_RTOL, "packed hn")
    assert_close(cn, z["cn"], LSTM_ATOL, LSTM_RTOL, "packed cn")


# (T, B, I, H, L, bidirectional, has_biases, batch_first, nonzero state)
CASES = [
    (1, 1, 8, 16, 1, False, True, False, True),
    (2, 1, 16, 48, 2, False, True, False, False),
    (3, 1, 8, 24, 1, False, True, False, True),
    (20, 1, 240, 128, 2, False, True, False, True),
    (16, 1, 64, 320, 2, False, True, False, True),      # prediction-net width
    (12, 1, 40, 1024, 1, False, True, False, True),
    (9, 1, 32, 64, 3, True, True, False, True),
    (10, 1, 32, 64, 2, False, False, True, False),
    (7, 5, 24, 48, 2, True, True, True, True),           # B > 1, bidirectional, batch_first
    (11, 8, 40, 128, 2, False, True, False, True),       # a full tile of sequences
    (6, 8, 240, 1024, 1, False, True, True, False),      # eight utterances at the encoder width
    (5, 11, 16, 32, 1, False, True, False, True),        # two tiles of sequences, the second ragged
    (9, 32, 64, 256, 2, False, True, True, True),        # four full tiles, batch_first
    (4, 19, 24, 1024, 1, True, True, False, True),       # ragged third tile, bidirectional, encoder width
    (3, 40, 16, 32, 1, False, True, False, True),        # eight tiles, the last ones ragged
    (5, 64, 240, 1024, 1, False, True, True, False),     # 64 utterances at the encoder width, batch_first
    (4, 57, 32, 128, 2, True, True, False, True),        # ragged eighth tile, bidirectional, two layers
    (2, 70, 16, 32, 1, False, True, False, True),        # 65..128 sequences: two batch halves, the second ragged
    (4, 128, 32, 1024, 1, False, True, True, False),     # the largest lock-step batch at the encoder width, batch_first
    (3, 97, 24, 256, 2, True, True, False, True),        # ragged second half, bidirectional, two layers
    (5, 33, 16, 1024, 1, False, True, False, True),      # smallest batch the pipelined kernel takes by default
    (3, 2, 7, 5, 2, False, True, False, True),           # odd sizes: scalar path
    (1, 8, 16, 32, 1, False, True, False, True),         # decode form, 8+ sequences: products as GEMMs + gate kernel
    (1, 33, 64, 128, 2, False, True, False, True),       # ... two layers, ragged row tiles
    (1, 128, 2048, 1024, 1, False, True, True, True),    # ... a GNMT decoder layer for 128 sentences
    (1, 20, 24, 48, 2, True, False, False, False),       # ... bidirectional, no biases, zero state
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("variant", ["streamed", "persistent", "pipe", "wide", "ksplit", "tagged"])
def test_lstm_matches_oracle(case, variant):
    ops = _ops()
    T, B, I, H, L, bi, hb, bf, nz = case
    if variant in ("persistent", "pipe") and (B > 128 or H % 16):
        pytest.skip("the persistent kernels take up to 128 sequences and H % 16 == 0")
    if variant == "wide" and (B > 64 or H % 16):
        pytest.skip("the exchange-on-compute-warps kernel takes up to 64 sequences and H % 16 == 0")
    if variant == "ksplit" and (B < 2 or B > 32 or H % 16):
        pytest.skip("the K-split batched kernel takes 2..32 sequences and H % 16 == 0")
    if variant == "tagged" and (B > 8 or H % 16):
        pytest.skip("tagged-word exchange takes up to 8 sequences and H % 16 == 0")
    D = 2 if bi else 1
    g = torch.Generator().manual_seed(T * 131 + H)
    ps = lstm_params(L, D, I, H, g, has_biases=hb)
    x = h16(torch.randn((B, T, I) if bf else (T, B, I), generator=g))
    h0 = h16(torch.randn(L * D, B, H, generator=g) * 0.5) if nz else None
    c0 = h16(torch.randn(L * D, B, H, generator=g) * 0.5) if nz else None
    ref = co.lstm(x.numpy(), [p.numpy() for p in ps], L, bi, hb, None if h0 is None else h0.numpy(),
                  None if c0 is None else c0.numpy(), bf)
    vid = {"streamed": ops.LSTM_STREAMED, "persistent": ops.LSTM_PERSISTENT, "pipe": ops.LSTM_PERSISTENT,
           "wide": ops.LSTM_PERSISTENT, "ksplit": ops.LSTM_PERSISTENT, "tagged": ops.LSTM_PERSISTENT_TAGGED}[variant]
    got = _run(ops, ps, x, h0, c0, L, bi, hb, bf, vid, bulk_wide={"ksplit": 0, "wide": 1, "pipe": 3}.get(variant))
    for name, a, b in zip(("y", "hn", "cn"), got, ref):
        assert_close(a, b, LSTM_ATOL, LSTM_RTOL, f"{variant} {name} {case}")


@pytest.mark.parametrize("variant", ["streamed", "persistent"])
def test_lstm_baseline_c1_vs_libtorch(variant):
    # C1: 2 layers, input 240, hidden 1024, T=200, B=1; x~N(0,1); params~U(-1/32,1/32); h0=c0=0; seed 0
    ops = _ops()
    torch.manual_seed(0)
    T, I, H, L = 200, 240, 1024, 2
    x = h16(torch.randn(T, 1, I))
    ps = []
    for l in range(L):
        Il = I if l == 0 else H
        ps += [h16((torch.rand(4 * H, Il) * 2 - 1) / 32), h16((torch.rand(4 * H, H) * 2 - 1) / 32),
               h16((torch.rand(4 * H) * 2 - 1) / 32), h16((torch.rand(4 * H) * 2 - 1) / 32)]
    z = torch.zeros(L, 1, H)
    y_ref, hn_ref, cn_ref = torch.lstm(x, [z, z], ps, True, L, 0.0, False, False, False)
    y, hn, cn = _run(ops, ps, x, None, None, L, False, True, False,
                     ops.LSTM_STREAMED if variant == "streamed" else ops.LSTM_PERSISTENT)
    assert_close(y, y_ref, CONTRACT_ATOL, CONTRACT_RTOL, "C1 y (contract)")
    e = assert_close(y, y_ref, LSTM_ATOL, LSTM_RTOL, "C1 y")
    assert_close(hn, hn_ref, LSTM_ATOL, LSTM_RTOL, "C1 hn")
    assert_close(cn, cn_ref, 2 * LSTM_ATOL, LSTM_RTOL, "C1 cn")
    print(f"C1 {variant}: max abs err {e:.2e}")


def test_lstm_variants_agree_and_repeat():
    # same handle, three calls in a row: step tags of the persistent exchange must not collide
    ops = _ops()
    g = torch.Generator().manual_seed(5)
    T, I, H, L = 33, 64, 256, 2
    ps = lstm_params(L, 1, I, H, g)
    x = h16(torch.randn(T, 1, I, generator=g))
    m = ops.Lstm([to_dev(p) for p in ps], L, False, I, H, True)
    m.set_variant(ops.LSTM_STREAMED)
    ys, hs, cs = m.forward(to_dev(x))
    m.set_variant(ops.LSTM_PERSISTENT)
    for _ in range(3):
        yp, hp, cp = m.forward(to_dev(x))
        torch.cuda.synchronize()
        assert m.last_status() == 0
        assert_close(yp, ys, 1e-3, 1e-3, "persistent vs streamed")
        assert_close(cp, cs, 2e-3, 1e-3, "persistent vs streamed cn")


def test_lstm_outputs_alias_slices_of_caller_buffers():
    # GNMT-style in-place "custom cat": y goes into the first half of a {1,1,2048} buffer, (h,c) into
    # slots of an {8,1,1024} state buffer (miopen_ops_executor.cpp:193-228)
    ops = _ops()
    g = torch.Generator().manual_seed(6)
    I = H = 1024
    ps = lstm_params(1, 1, I, H, g)
    x = h16(torch.randn(1, 1, I, generator=g))
    h0 = h16(torch.randn(1, 1, H, generator=g) * 0.5)
    c0 = h16(torch.randn(1, 1, H, generator=g) * 0.5)
    ref = co.lstm(x.numpy(), [p.numpy() for p in ps], 1, False, True, h0.numpy(), c0.numpy())
    cat_buf = torch.full((1, 1, 2048), 5.0, dtype=torch.float16, device="cuda")
    state_buf = torch.full((8, 1, 1024), 5.0, dtype=torch.float16, device="cuda")
    m = ops.Lstm([to_dev(p) for p in ps], 1, False, I, H, True)
    m.forward(to_dev(x), to_dev(h0), to_dev(c0), out=(cat_buf[..., :1024], state_buf[2:3], state_buf[3:4]))
    torch.cuda.synchronize()
    assert_close(cat_buf[..., :1024], ref[0], LSTM_ATOL, LSTM_RTOL, "aliased y")
    assert_close(state_buf[2:3], ref[1], LSTM_ATOL, LSTM_RTOL, "aliased hn")
    assert_close(state_buf[3:4], ref[2], LSTM_ATOL, LSTM_RTOL, "aliased cn")
    assert (cat_buf[..., 1024:] == 5).all() and (state_buf[:2] == 5).all() and (state_buf[4:] == 5).all()


@pytest.mark.parametrize("B,L", [(1, 1), (4, 1), (40, 1), (2, 2), (150, 1)])
def test_persistent_bounded_wait_reports_timeout_and_context_survives(B, L):
    # Fault handling without faulting anything: shrink the bounded wait to a single poll, so the hidden-state exchange
    # cannot complete in time; the kernel must give up, record ERR_TIMEOUT and return, and the next call (normal
    # limit) must still be correct.  L = 2 with two sequences is a layer wavefront.
    ops = _ops()
    from pimaicompiler_b200 import _lib
    g = torch.Generator().manual_seed(17)
    T, I, H = 64, 32, 256
    ps = lstm_params(L, 1, I, H, g)
    x = h16(torch.randn(T, B, I, generator=g))
    m = ops.Lstm([to_dev(p) for p in ps], L, False, I, H, True)
    m.set_variant(ops.LSTM_PERSISTENT)
    lib = _lib.lib()
    assert lib.pimb200_lstm_set_poll_limit(m._h, 1) == 0
    m.forward(to_dev(x))
    torch.cuda.synchronize()                      # returns: nothing hangs
    assert m.last_status() == _lib.ERR_TIMEOUT
    assert m.last_status() == 0                   # reading clears it
    assert lib.pimb200_lstm_set_poll_limit(m._h, 1 << 21) == 0
    y, hn, cn = m.forward(to_dev(x))
    torch.cuda.synchronize()
    assert m.last_status() == 0
    ref = co.lstm(x.numpy(), [p.numpy() for p in ps], L, False)
    assert_close(y, ref[0], LSTM_ATOL, LSTM_RTOL, "after a timed-out launch")
    # a timed-out launch must not poison the launches behind it: nobody reads (and thereby clears) the status between
    # the two calls here, the second call must be correct all the same, and the time-out is still reported afterwards
    assert lib.pimb200_lstm_set_poll_limit(m._h, 1) == 0
    m.forward(to_dev(x))
    assert lib.pimb200_lstm_set_poll_limit(m._h, 1 << 21) == 0
    y2, _, _ = m.forward(to_dev(x))
    torch.cuda.synchronize()
    assert_close(y2, ref[0], LSTM_ATOL, LSTM_RTOL, "directly behind a timed-out launch, status unread")
    assert m.last_status() == _lib.ERR_TIMEOUT


@pytest.mark.parametrize("B,L,H", [(1, 1, 1024), (8, 1, 320), (16, 1, 1024), (1, 2, 1024), (8, 2, 256), (20, 1, 1024), (64, 1, 320),
                                   (70, 1, 256), (128, 1, 1024), (300, 1, 1024), (200, 1, 320)])
def test_waits_that_run_out_in_different_steps(B, L, H):
    # limits of a few polls, which some warps of a CTA reach a step or two before others: every launch returns, a launch that
    # lost a wait says so, one that did not is right, and so is the next one with the normal limit
    ops = _ops()
    from pimaicompiler_b200 import _lib
    g = torch.Generator().manual_seed(B + L)
    T, I = 64, 32
    ps = lstm_params(L, 1, I, H, g)
    x = h16(torch.randn(T, B, I, generator=g))
    m = ops.Lstm([to_dev(p) for p in ps], L, False, I, H, True)
    m.set_variant(ops.LSTM_PERSISTENT)
    want = [t.clone() for t in m.forward(to_dev(x))]
    lost = 0
    for limit in (2, 2, 3, 3, 4, 4, 6, 8, 16):
        assert _lib.lib().pimb200_lstm_set_poll_limit(m._h, limit) == 0
        got = m.forward(to_dev(x))
        torch.cuda.synchronize()
        status = m.last_status()
        assert status in (0, _lib.ERR_TIMEOUT)
        lost += status != 0
        assert status != 0 or all(torch.equal(a, b) for a, b in zip(got, want))
        assert _lib.lib().pimb200_lstm_set_poll_limit(m._h, 1 << 21) == 0
        got = m.forward(to_dev(x))
        torch.cuda.synchronize()
        assert m.last_status() == 0
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert lost > 0                               # (a limit of two is too few for a launch's first step)


@pytest.mark.parametrize("H", [48, 320, 1024])
@pytest.mark.parametrize("B,L", [(1, 1), (3, 2), (8, 2), (9, 1), (15, 1), (16, 1), (17, 1), (32, 1), (33, 1), (49, 1), (65, 1), (96, 1), (97, 1)])
def test_recurrence_kernels_at_the_edges_of_their_ranges(B, L, H):
    # batch sizes where the choice of kernel, its groups or its halves change; more steps than the exchange has buffers;
    # a sequence of NaNs (the exchange's marker for "not written yet" is one) must leave the others alone
    ops = _ops()
    g = torch.Generator().manual_seed(B * 11 + H)
    T, I = 11, 24
    ps = lstm_params(L, 1, I, H, g)
    x = h16(torch.randn(T, B, I, generator=g))
    h0, c0 = (h16(torch.randn(L, B, H, generator=g) * 0.5) for _ in range(2))
    ref = co.lstm(x.numpy(), [p.numpy() for p in ps], L, False, True, h0.numpy(), c0.numpy(), False)
    got = _run(ops, ps, x, h0, c0, L, False, True, False, ops.LSTM_PERSISTENT)
    for name, a, b in zip(("y", "hn", "cn"), got, ref):
        assert_close(a, b, LSTM_ATOL, LSTM_RTOL, f"{name} B {B} H {H}")
    if B > 1:
        x[3, 1] = float("nan")
        y = _run(ops, ps, x, h0, c0, L, False, True, False, ops.LSTM_PERSISTENT)[0].cpu()
        assert torch.isnan(y[3:, 1]).all()
        keep = [b for b in range(B) if b != 1]
        assert_close(y[:, keep], ref[0][:, keep], LSTM_ATOL, LSTM_RTOL, f"beside a NaN sequence, B {B} H {H}")


@pytest.mark.parametrize("B,L", [(3, 2), (8, 2), (3, 1), (9, 1), (20, 1), (70, 1)])
def test_initial_state_of_nans_with_every_bit_set(B, L):
    _nan_state(B, L, 256)


@pytest.mark.parametrize("B", [70, 128])
def test_initial_state_of_nans_in_two_halves_of_a_large_layer(B):
    _nan_state(B, 1, 1024)


def _nan_state(B, L, H):
    # 0xffff is a NaN and the exchange's mark of a record that has not arrived
    ops = _ops()
    g = torch.Generator().manual_seed(B)
    T, I = 12, 24
    m = ops.Lstm([to_dev(p) for p in lstm_params(L, 1, I, H, g)], L, False, I, H, True)
    x, h0, c0 = (to_dev(torch.randn(*s, generator=g)) for s in ((T, B, I), (L, B, H), (L, B, H)))
    want = [t.clone() for t in m.forward(x, h0, c0)]
    h0.view(torch.int16)[L - 1, 1] = -1
    got = m.forward(x, h0, c0)
    torch.cuda.synchronize()
    assert m.last_status() == 0
    assert torch.isnan(got[0][:, 1]).all() and torch.isnan(got[1][L - 1, 1]).all()
    keep = [b for b in range(B) if b != 1]
    assert all(torch.equal(a[:, keep], b[:, keep]) for a, b in zip(got, want))


@pytest.mark.parametrize("L,B,T", [(1, 1, 10), (1, 1, 11), (1, 8, 12), (1, 16, 13), (2, 1, 8), (2, 3, 9), (2, 8, 10), (3, 2, 11),
                                   (1, 20, 8), (1, 40, 10), (2, 70, 11), (1, 128, 9)])
def test_captured_recurrence_replayed_among_eager_calls(L, B, T):
    _captured_among_eager_calls(L, B, T, 256)


@pytest.mark.parametrize("L,B,T", [(2, 70, 11), (1, 128, 9)])
def test_captured_recurrence_of_a_large_layer(L, B, T):
    # 65..128 sequences of 1024 units: the pipelined kernel in two halves
    _captured_among_eager_calls(L, B, T, 1024)


def _captured_among_eager_calls(L, B, T, H):
    # a call that was captured and never run, and replays of graphs with one, two or three recurrences of a handle between
    # eager calls: always what a handle of its own gives, bit for bit
    ops = _ops()
    g = torch.Generator().manual_seed(L * 100 + B)
    I = 24
    ps = [to_dev(p) for p in lstm_params(L, 1, I, H, g)]
    m = ops.Lstm(ps, L, False, I, H, True)
    xs = [to_dev(torch.randn(T, B, I, generator=g)) for _ in range(7)]
    want = [[t.clone() for t in ops.Lstm(ps, L, False, I, H, True).forward(x)] for x in xs]

    def check(i, got):
        torch.cuda.synchronize()
        assert m.last_status() == 0
        assert all(torch.equal(a, b) for a, b in zip(got, want[i])), f"input {i}"

    check(0, m.forward(xs[0]))                                   # (workspaces grow outside a capture)
    x = xs[1].clone()
    graphs = []
    for calls in (1, 2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(calls):
                got = m.forward(x)
        graphs.append((graph, got))
        check(2, m.forward(xs[2]))
    for i in (3, 4, 5, 6, 0, 1):
        for graph, got in graphs:
            x.copy_(xs[i])
            graph.replay()
            check(i, got)
        if i % 2:
            check(i - 1, m.forward(xs[i - 1]))


@pytest.mark.parametrize("bulk_wide", [1, 3])
@pytest.mark.parametrize("L", [1, 2])
def test_a_chosen_recurrence_kernel_runs_at_every_batch_size(bulk_wide, L):
    # within one kernel a sequence's result does not depend on how many share the launch; another kernel sums in another order
    ops = _ops()
    g = torch.Generator().manual_seed(L)
    T, I, H = 40, 24, 1024
    ps = lstm_params(L, 1, I, H, g)
    x = h16(torch.randn(T, 32, I, generator=g))
    run = lambda b, bw: [t.clone() for t in _run(ops, ps, x[:, :b], None, None, L, False, True, False, ops.LSTM_AUTO, bw)]  # noqa: E731
    many = run(32, bulk_wide)
    for b in (1, 4, 16):
        assert all(torch.equal(f, m[:, :b]) for f, m in zip(run(b, bulk_wide), many)), f"{b} sequences"
    assert not torch.equal(run(4, None)[0], many[0][:, :4])          # (the default kernel's differ, so the above means something)


@pytest.mark.parametrize("T,B,I,H", [(6, 64, 64, 1024), (9, 23, 32, 256), (5, 40, 16, 128)])
def test_tcgen05_recurrence_variant_matches_oracle(T, B, I, H):
    # the opt-in tensor-memory variant of the batched recurrence must give the same results as the default kernels
    ops = _ops()
    from pimaicompiler_b200 import _lib
    g = torch.Generator().manual_seed(B * 7 + H)
    ps = lstm_params(1, 1, I, H, g)
    x = h16(torch.randn(T, B, I, generator=g))
    h0 = h16(torch.randn(1, B, H, generator=g) * 0.5)
    c0 = h16(torch.randn(1, B, H, generator=g) * 0.5)
    ref = co.lstm(x.numpy(), [p.numpy() for p in ps], 1, False, True, h0.numpy(), c0.numpy())
    m = ops.Lstm([to_dev(p) for p in ps], 1, False, I, H, True)
    m.set_variant(ops.LSTM_PERSISTENT)
    assert _lib.lib().pimb200_lstm_set_use_tc(m._h, 1) == 0
    got = m.forward(to_dev(x), to_dev(h0), to_dev(c0))
    torch.cuda.synchronize()
    assert m.last_status() == 0
    for name, a, b in zip(("y", "hn", "cn"), got, ref):
        assert_close(a, b, LSTM_ATOL, LSTM_RTOL, f"tcgen05 recurrence {name}")


def test_lstm_benchmark_shape_batched_properties():
    # the benchmark's pre-net shape at full size: 64 sequences x 1000 steps, batch-first (the projection is then written
    # time-major through the 3-D tensor map).  Size-independent properties instead of an oracle run:
    #   * the persistent kernel agrees with the streamed one (different kernels, different summation order);
    #   * a repeat is bit-identical;
    #   * every sequence is computed independently of its batch: a sub-batch reproduces its rows bit for bit
    ops = _ops()
    g = torch.Generator().manual_seed(64)
    T, B, I, H, L = 1000, 64, 240, 1024, 2
    ps = [to_dev(p) for p in lstm_params(L, 1, I, H, g, scale=1 / 32)]
    x = to_dev(h16(torch.randn(B, T, I, generator=g)))
    m = ops.Lstm(ps, L, False, I, H, True)
    m.set_variant(ops.LSTM_PERSISTENT)
    y, hn, cn = m.forward(x, batch_first=True)
    y2, hn2, cn2 = m.forward(x, batch_first=True)
    torch.cuda.synchronize()
    assert m.last_status() == 0
    assert torch.equal(y, y2) and torch.equal(hn, hn2) and torch.equal(cn, cn2)
    assert torch.isfinite(y.float()).all()
    m.set_variant(ops.LSTM_STREAMED)
    ys, hns, cns = m.forward(x, batch_first=True)
    assert_close(y, ys, LSTM_ATOL, LSTM_RTOL, "persistent vs streamed y at T=1000, B=64")
    assert_close(cn, cns, LSTM_ATOL, LSTM_RTOL, "persistent vs streamed c_n")
    m.set_variant(ops.LSTM_PERSISTENT)
    # a smaller lock-step batch of the same kernel (17..128 sequences) reproduces its rows bit for bit
    yb, hnb, cnb = m.forward(x[20:60].contiguous(), batch_first=True)
    assert torch.equal(yb, y[20:60]) and torch.equal(hnb, hn[:, 20:60]) and torch.equal(cnb, cn[:, 20:60])
    yw, hnw, cnw = m.forward(x[20:44].contiguous(), batch_first=True)
    assert torch.equal(yw, y[20:44]) and torch.equal(hnw, hn[:, 20:44]) and torch.equal(cnw, cn[:, 20:44])
    # 16 sequences or fewer run on the few-sequence kernel (another summation order): within the tolerance
    yw, hnw, cnw = m.forward(x[20:32].contiguous(), batch_first=True)
    assert_close(yw, y[20:32], LSTM_ATOL, LSTM_RTOL, "12 sequences alone vs in the batch of 64")
    # a single sequence runs on the low-latency kernel (another summation order): equal within the LSTM tolerance
    for n in (0, 37, 63):
        y1, hn1, cn1 = m.forward(x[n:n + 1].contiguous(), batch_first=True)
        assert_close(y1[0], y[n], LSTM_ATOL, LSTM_RTOL, f"sequence {n} alone vs in the batch")
        assert_close(cn1[:, 0], cn[:, n], LSTM_ATOL, LSTM_RTOL, f"c_n of sequence {n} alone vs in the batch")


def test_lstm_benchmark_shape_batched_vs_libtorch():
    # the benchmark's pre-net recurrence at full size (2 layers, 240 -> 1024, 1000 steps, 64 sequences in lock step,
    # batch-first) against live libtorch CPU fp32 for three of the 64 sequences: the whole output sequence, h_n and c_n.
    # fp16 hidden states feed back through 1000 steps here; the error at the last step is printed.
    ops = _ops()
    g = torch.Generator().manual_seed(65)
    T, B, I, H, L = 1000, 64, 240, 1024, 2
    ps = lstm_params(L, 1, I, H, g, scale=1 / 32)
    x = h16(torch.randn(B, T, I, generator=g))
    m = ops.Lstm([to_dev(p) for p in ps], L, False, I, H, True)
    y, hn, cn = m.forward(to_dev(x), batch_first=True)
    torch.cuda.synchronize()
    assert m.last_status() == 0
    z = torch.zeros(L, 1, H)
    for n in (0, 21, 63):
        with torch.no_grad():
            yr, hr, cr = torch.lstm(x[n:n + 1], [z, z], ps, True, L, 0.0, False, False, True)
        e = assert_close(y[n], yr[0], CONTRACT_ATOL, CONTRACT_RTOL, f"y of sequence {n} at T=1000, B=64")
        e_last = float((y[n, -1].float().cpu() - yr[0, -1]).abs().max())
        assert_close(hn[:, n], hr[:, 0], CONTRACT_ATOL, CONTRACT_RTOL, f"h_n of sequence {n}")
        assert_close(cn[:, n], cr[:, 0], CONTRACT_ATOL, CONTRACT_RTOL, f"c_n of sequence {n}")
        print(f"sequence {n}: max err over 1000 steps {e:.2e}, at the last step {e_last:.2e}")


@pytest.mark.parametrize("B,I,H,L,bi,lo,hi", [(7, 24, 64, 2, True, 1, 9), (40, 1024, 1024, 1, True, 20, 50), (128, 48, 128, 2, False, 3, 30),
                                             (33, 40, 256, 3, True, 2, 12), (5, 16, 48, 1, False, 4, 4),
                                             (96, 64, 1024, 1, True, 8, 20), (200, 40, 256, 2, True, 3, 14), (300, 24, 320, 2, False, 5, 20)])
def test_lstm_packed_sequences_on_the_lockstep_kernels_vs_libtorch(B, I, H, L, bi, lo, hi):
    # packed input (sequences of ragged length, sorted) runs as a padded lock-step batch on the persistent recurrences:
    # outputs, h_n and c_n against libtorch's packed overload, and against the timestep-by-timestep streamed path
    ops = _ops()
    g = torch.Generator().manual_seed(B * 7 + H)
    D = 2 if bi else 1
    lens = sorted((int(v) for v in torch.randint(lo, hi + 1, (B,), generator=g)), reverse=True)
    T = lens[0]
    ps = lstm_params(L, D, I, H, g)
    x = h16(torch.randn(T, B, I, generator=g))
    h0 = h16(torch.randn(L * D, B, H, generator=g) * 0.5)
    c0 = h16(torch.randn(L * D, B, H, generator=g) * 0.5)
    packed = torch.nn.utils.rnn.pack_padded_sequence(x, torch.tensor(lens), enforce_sorted=True)
    with torch.backends.mkldnn.flags(enabled=False):
        ry, rhn, rcn = torch.lstm(packed.data, packed.batch_sizes, [h0, c0], ps, True, L, 0.0, False, bi)
    m = ops.Lstm([to_dev(p) for p in ps], L, bi, I, H, True)
    y, hn, cn = m.forward_packed(to_dev(packed.data), packed.batch_sizes, to_dev(h0), to_dev(c0))
    assert m.last_status() == 0
    assert_close(y, ry, LSTM_ATOL, LSTM_RTOL, "packed y on the lock-step kernels")
    assert_close(hn, rhn, LSTM_ATOL, LSTM_RTOL, "packed h_n")
    assert_close(cn, rcn, LSTM_ATOL, LSTM_RTOL, "packed c_n")
    m.set_packed_lockstep(False)
    ys, hns, cns = m.forward_packed(to_dev(packed.data), packed.batch_sizes, to_dev(h0), to_dev(c0))
    assert_close(ys, ry, LSTM_ATOL, LSTM_RTOL, "packed y, streamed")
    assert_close(y, ys, LSTM_ATOL, LSTM_RTOL, "lock-step vs streamed")
    assert_close(cn, cns, LSTM_ATOL, LSTM_RTOL, "lock-step vs streamed c_n")


@pytest.mark.parametrize("B,I,H", [(8, 64, 32), (33, 256, 128), (128, 2048, 1024), (96, 512, 320), (97, 96, 320), (64, 2048, 512), (65, 240, 64)])
def test_lstm_decode_step_with_strided_rows_and_residual(B, I, H):
    # the decode step that writes into one half of the next cell's concatenated input: equal to forward() with T = 1 bit
    # for bit, and to the fp16 add of a residual row
    ops = _ops()
    g = torch.Generator().manual_seed(B + I + H)
    ps = [to_dev(p) for p in lstm_params(1, 1, I, H, g)]
    m = ops.Lstm(ps, 1, False, I, H, True)
    xbuf = to_dev(h16(torch.randn(B, I + 24, generator=g)))          # the input is the first I columns of wider rows
    h0 = to_dev(h16(torch.randn(1, B, H, generator=g) * 0.5))
    c0 = to_dev(h16(torch.randn(1, B, H, generator=g) * 0.5))
    res = to_dev(h16(torch.randn(B, 2 * H, generator=g)))
    y_ref, hn_ref, cn_ref = m.forward(xbuf[:, :I].contiguous().view(1, B, I), h0, c0)
    out = torch.zeros(B, 2 * H, dtype=torch.float16, device="cuda")
    hn, cn = torch.empty(B, H, dtype=torch.float16, device="cuda"), torch.empty(B, H, dtype=torch.float16, device="cuda")
    assert m.forward_step(xbuf[:, :I], h0[0], c0[0], out[:, H:], hn, cn)
    assert torch.equal(out[:, H:], y_ref[0]) and torch.equal(hn, hn_ref[0]) and torch.equal(cn, cn_ref[0])
    assert float(out[:, :H].abs().max()) == 0.0
    assert m.forward_step(xbuf[:, :I], h0[0], c0[0], out[:, :H], hn, cn, residual=res[:, H:])
    assert torch.equal(out[:, :H], ops.add_f16(y_ref[0].contiguous(), res[:, H:].contiguous()))
    assert torch.equal(hn, hn_ref[0])
    small = ops.Lstm(ps, 1, False, I, H, True)
    assert not small.forward_step(xbuf[:4, :I], h0[0, :4].contiguous(), c0[0, :4].contiguous(), out[:4, :H], hn[:4], cn[:4])


@pytest.mark.parametrize("T,B,I,H,L,bf", [(20, 1, 240, 128, 2, False), (9, 3, 24, 64, 3, True), (12, 8, 40, 256, 4, False),
                                          (1000, 1, 240, 1024, 2, False), (33, 2, 2048, 1024, 3, False)])
def test_lstm_layer_wavefront_matches_oracle_and_sequential_layers(T, B, I, H, L, bf):
    # stacked layers of up to 8 sequences run in pairs, one step apart, in one launch (the batch-1 latency path): against
    # the C oracle, and against the same handle with the layers run one after the other
    ops = _ops()
    g = torch.Generator().manual_seed(T * 7 + H + L)
    ps = lstm_params(L, 1, I, H, g, scale=1 / 32 if H >= 1024 else None)
    x = h16(torch.randn((B, T, I) if bf else (T, B, I), generator=g))
    h0 = h16(torch.randn(L, B, H, generator=g) * 0.5)
    c0 = h16(torch.randn(L, B, H, generator=g) * 0.5)
    m = ops.Lstm([to_dev(p) for p in ps], L, False, I, H, True)
    y, hn, cn = m.forward(to_dev(x), to_dev(h0), to_dev(c0), batch_first=bf)
    y_again, _, _ = m.forward(to_dev(x), to_dev(h0), to_dev(c0), batch_first=bf)
    assert m.last_status() == 0 and torch.equal(y, y_again)
    m.set_wavefront(False)
    ys, hns, cns = m.forward(to_dev(x), to_dev(h0), to_dev(c0), batch_first=bf)
    assert_close(y, ys, LSTM_ATOL, LSTM_RTOL, "wavefront vs layer after layer: y")
    assert_close(hn, hns, LSTM_ATOL, LSTM_RTOL, "wavefront vs layer after layer: h_n")
    assert_close(cn, cns, LSTM_ATOL, LSTM_RTOL, "wavefront vs layer after layer: c_n")
    if T <= 40:
        ref = co.lstm(x.numpy(), [p.numpy() for p in ps], L, False, True, h0.numpy(), c0.numpy(), bf)
        for name, a, b in zip(("y", "hn", "cn"), (y, hn, cn), ref):
            assert_close(a, b, LSTM_ATOL, LSTM_RTOL, f"wavefront {name}")


def _libtorch(ps, x, h0, c0, L, bi, bf):
    state = tuple(torch.zeros(L * (2 if bi else 1), x.shape[0 if bf else 1], ps[1].shape[1]) if s is None else s for s in (h0, c0))
    return torch.lstm(x, state, ps, True, L, 0.0, False, bi, bf)


# (T, B, I, H, L, bidirectional, batch_first, state): sub-batches of every width of the tensor-core recurrence (16 columns a step
# at H = 1024: four groups of two), one sub-batch per group, several parts, several chunks of steps, a ragged last group
@pytest.mark.parametrize("T,B,I,H,L,bi,bf,state", [
    (8, 129, 24, 1024, 1, False, False, True), (9, 257, 8, 1024, 1, False, False, False), (8, 512, 8, 1024, 1, False, True, True),
    (8, 520, 8, 1024, 1, False, False, True), (8, 700, 8, 1024, 1, False, False, True), (10, 897, 8, 1024, 1, False, False, True),
    (8, 1025, 16, 1024, 1, False, False, True), (11, 150, 20, 320, 3, False, True, True), (12, 200, 64, 512, 2, True, True, True),
    (9, 260, 64, 960, 1, True, False, True), (8, 130, 7, 64, 2, True, False, False), (130, 1024, 8, 64, 1, False, False, True),
    (70, 1030, 8, 64, 1, True, True, True)])
def test_many_sequences_on_the_tensor_core_recurrence_vs_libtorch(T, B, I, H, L, bi, bf, state):
    ops = _ops()
    g = torch.Generator().manual_seed(T * B + H)
    ps = lstm_params(L, 2 if bi else 1, I, H, g)
    x = h16(torch.randn(*((B, T, I) if bf else (T, B, I)), generator=g))
    LD = L * (2 if bi else 1)
    h0, c0 = (h16(torch.randn(LD, B, H, generator=g) * 0.5) for _ in range(2)) if state else (None, None)
    y, hn, cn = _run(ops, ps, x, h0, c0, L, bi, True, bf, ops.LSTM_AUTO)
    ref = _libtorch(ps, x, h0, c0, L, bi, bf)
    for got, want, name in zip((y, hn, cn), ref, ("y", "hn", "cn")):
        assert_close(got, want.numpy(), LSTM_ATOL, LSTM_RTOL, name)


@pytest.mark.parametrize("B,H,bi", [(3, 64, False), (20, 64, False), (40, 64, True), (70, 256, False), (150, 256, False)])
def test_packed_sequences_end_under_products_of_any_size(B, H, bi):
    # recurrent weights whose products are far beyond the range of a gate: behind a sequence's end nothing reaches its cell state
    ops = _ops()
    g = torch.Generator().manual_seed(B)
    T, I, D = 12, 16, 2 if bi else 1
    ps = lstm_params(1, D, I, H, g)
    for d in range(D):
        ps[4 * d] = h16(ps[4 * d].abs() * 4)                         # positive states: gates fully open, c grows by one a step
        ps[4 * d + 1] = torch.full((4 * H, H), 1000.0)
    x = h16(torch.rand(T, B, I, generator=g) + 0.5)
    lens = torch.randint(1, T + 1, (B,), generator=g).sort(descending=True).values
    lens[0] = T
    packed = torch.nn.utils.rnn.pack_padded_sequence(x, lens)
    zero = torch.zeros(D, B, H)
    with torch.backends.mkldnn.flags(enabled=False):
        ref = torch.lstm(packed.data, packed.batch_sizes, [zero, zero], ps, True, 1, 0.0, False, bi)
    assert float(ref[2].min()) < T - 3 and float(ref[2].max()) > T - 1
    m = ops.Lstm([to_dev(p) for p in ps], 1, bi, I, H, True)
    got = m.forward_packed(to_dev(packed.data), packed.batch_sizes)
    torch.cuda.synchronize()
    assert m.last_status() == 0
    for a, b, name in zip(got, ref, ("y", "hn", "cn")):
        assert_close(a, b.numpy(), LSTM_ATOL, LSTM_RTOL, name)


# (T, B, H, bidirectional, packed, MiB left): the recurrence for many sequences wants the gate terms of both directions, or padded
# rows, where the kernels before it take one direction, or packed rows
@pytest.mark.parametrize("T,B,H,bi,packed,left", [(400, 96, 1024, True, True, 1024), (300, 150, 1024, True, False, 1100)])
def test_smaller_workspaces_where_memory_is_short(T, B, H, bi, packed, left):
    ops = _ops()
    g = torch.Generator().manual_seed(B)
    I, D = 64, 2 if bi else 1
    ps = [to_dev(p) for p in lstm_params(1, D, I, H, g)]
    lens = torch.linspace(T, T // 2, B).long()
    sizes = (lens[:, None] > torch.arange(T)).sum(0)
    x = to_dev(torch.randn(*((int(sizes.sum()), I) if packed else (T, B, I)), generator=g))
    call = (lambda m: m.forward_packed(x, sizes)) if packed else (lambda m: m.forward(x))
    want = [t.clone() for t in call(ops.Lstm(ps, 1, bi, I, H, True))]
    m = ops.Lstm(ps, 1, bi, I, H, True)
    with device_memory_left(left << 20):
        out = call(m)
        torch.cuda.synchronize()
    assert m.last_status() == 0
    for got, ref, name in zip(out, want, ("y", "hn", "cn")):
        assert_close(got, ref.float().cpu().numpy(), LSTM_ATOL, LSTM_RTOL, name)
    for got, ref in zip(call(m), want):                       # and with room again
        assert torch.equal(got, ref)


@pytest.mark.parametrize("sizes", [((1024, 150), (320, 520)), ((1024, 40), (256, 40)), ((1024, 1), (64, 1))])
def test_threads_with_handles_of_different_sizes_launch_the_same_kernel(sizes):
    # the same instance with different amounts of shared memory, whose limit belongs to the kernel: no thread takes it from another
    import threading
    ops = _ops()
    from pimaicompiler_b200 import _lib
    g = torch.Generator().manual_seed(5)
    T, I, jobs, failed = 8, 24, [], []
    for H, B in sizes:
        m = ops.Lstm([to_dev(p) for p in lstm_params(1, 1, I, H, g)], 1, False, I, H, True)
        x = to_dev(torch.randn(T, B, I, generator=g))
        want = m.forward(x)[0].clone()
        jobs.append((m, x, torch.empty_like(want), want))
    stream = torch.cuda.Stream()               # one for both: the threads meet on the host only
    torch.cuda.synchronize()

    def loop(m, x, y, want):
        torch.cuda.set_device(0)
        for _ in range(150):
            if rc := _lib.lib().pimb200_lstm_forward(m._h, x.data_ptr(), T, x.shape[1], None, None, y.data_ptr(), None, None, 0, stream.cuda_stream):
                failed.append(rc)

    threads = [threading.Thread(target=loop, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    torch.cuda.synchronize()
    for m, _, y, want in jobs:
        assert m.last_status() == 0 and torch.equal(y, want)


@pytest.mark.parametrize("H,B", [(320, 224), (512, 100), (64, 40), (1024, 300)])
def test_trace_buffer_of_one_record_per_eight_units_is_not_overrun(H, B):
    # the recurrence for many sequences has up to 148 CTAs at any hidden size; the buffer has room for H / 8
    ops = _ops()
    from pimaicompiler_b200 import _lib
    g = torch.Generator().manual_seed(H)
    T, I, bi = 9, 24, B == 40
    m = ops.Lstm([to_dev(p) for p in lstm_params(1, 2 if bi else 1, I, H, g)], 1, bi, I, H, True)
    words, guard = -(-H // 8) * T * 8, 148 * T * 8
    trace = torch.full((words + guard,), -1, dtype=torch.int64, device="cuda")
    assert _lib.lib().pimb200_lstm_set_trace(m._h, trace.data_ptr()) == 0
    m.forward(to_dev(torch.randn(T, B, I, generator=g)))
    torch.cuda.synchronize()
    assert _lib.lib().pimb200_lstm_set_trace(m._h, None) == 0
    assert bool((trace[words:] == -1).all()) and bool((trace[:words] != -1).any())


def test_outputs_given_in_any_sequence_and_batch_sizes_of_any_array():
    ops = _ops()
    g = torch.Generator().manual_seed(2)
    T, B, I, H = 4, 3, 16, 32
    m = ops.Lstm([to_dev(p) for p in lstm_params(1, 1, I, H, g)], 1, False, I, H, True)
    x = to_dev(torch.randn(T, B, I, generator=g))
    want = m.forward(x)
    fresh = lambda: [torch.empty_like(t) for t in want]  # noqa: E731
    for given in (tuple, list, iter, lambda ts: (t for t in ts)):
        ts = fresh()
        got = m.forward(x, out=given(ts))
        assert isinstance(got, tuple) and all(a is b for a, b in zip(got, ts))
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    y, hn, cn = fresh()
    assert m.forward(x, out=(y, None, None)) == (y, None, None) and torch.equal(y, want[0])
    for wrong in ((y, 5, cn), (y, hn), (y, "cn", None)):
        with pytest.raises(Exception):
            m.forward(x, out=wrong)
    data = to_dev(torch.randn(7, I, generator=g))
    sizes = np.array([3, 2, 2])
    want = m.forward_packed(data, torch.from_numpy(sizes))
    for given in (sizes, sizes.astype(np.int32), torch.from_numpy(sizes).int(), torch.from_numpy(sizes).cuda(), torch.from_numpy(sizes).float()):
        assert all(torch.equal(a, b) for a, b in zip(m.forward_packed(data, given), want))


@pytest.mark.parametrize("B,H", [(8, 1024), (32, 1024), (130, 512), (2048, 1024)])
def test_decode_step_whose_output_lies_over_its_input(B, H):
    ops = _ops()
    g = torch.Generator().manual_seed(B)
    I = H
    m = ops.Lstm([to_dev(p) for p in lstm_params(1, 1, I, H, g)], 1, False, I, H, True)
    rows = to_dev(torch.randn(B, 2 * H, generator=g))
    h0, c0 = (to_dev(torch.randn(B, H, generator=g) * 0.5) for _ in range(2))
    y, hn, cn = (torch.empty(B, H, dtype=torch.float16, device="cuda") for _ in range(3))
    assert m.forward_step(rows[:, :I], h0, c0, y, hn, cn)
    for _ in range(10):
        for at in (0, 8, H // 2, H):                # H: the other half of the same rows, which overlaps nothing
            buf, hb, cb = rows.clone(), torch.empty_like(hn), torch.empty_like(cn)
            assert m.forward_step(buf[:, :I], h0, c0, buf[:, at:at + H], hb, cb)
            for got, want in ((buf[:, at:at + H], y), (hb, hn), (cb, cn)):
                assert_close(got, want, LSTM_ATOL, LSTM_RTOL, f"output {at} columns behind the input")
