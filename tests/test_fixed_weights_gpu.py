"""GPU: products whose weights nobody writes, which a launch may read before the work ahead of it has ended."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one and two 32-wide K blocks per warp, more than a warp's registers hold at once, ragged K, 16 and 32 weight rows per CTA, a warp
# per row tile, the tensor-core kernel, the SIMT one
@pytest.mark.parametrize("N,K,J", [(512, 512, 20), (512, 2048, 5), (1536, 512, 32), (2048, 512, 100), (32320, 512, 20), (4096, 1024, 500), (40, 72, 3), (512, 256, 9), (2048, 520, 17), (512, 1024, 33), (100, 63, 5)])
def test_products_with_fixed_weights(N, K, J):
    from pimaicompiler_b200 import ops
    ops.init()
    g = torch.Generator(device="cuda").manual_seed(N + K + J)
    W, X, b = (torch.randn(*s, generator=g, device="cuda").half() for s in ((N, K), (J, K), (N,)))
    want = ops.gemm_wx(W, X, b, ops.ACT_RELU)
    for _ in range(3):                                          # behind one another: launches overlap their predecessors
        assert torch.equal(ops.gemm_wx_fixed(W, X, b, ops.ACT_RELU), want)
    assert torch.equal(ops.gemm_wx_fixed(W, X, b, ops.ACT_RELU, out_f32=True), ops.gemm_wx(W, X, b, ops.ACT_RELU, out_f32=True))


def _written(ops, g, shape, rows):
    """`rows` sources whose product writes a matrix or vector of the shape, and the call that writes it: a launch that lets the
    launches behind it start early."""
    n = shape[-1]
    P = torch.randn(n, 64, generator=g, device="cuda").half() * 0.125
    out = torch.empty(*shape, dtype=torch.float16, device="cuda")
    if len(shape) == 1:
        src = torch.randn(rows, 64, generator=g, device="cuda").half()
        return out, lambda i: ops.gemv_mv(P, src[i], None, out=out)
    src = torch.randn(rows, shape[0], 64, generator=g, device="cuda").half()
    return out, lambda i: ops.gemm_wx(P, src[i], None, out=out)


def _chained(call, writers, passes):
    """The results of `call` behind the writers, pass after pass without and with a wait in between."""
    got = []
    for i in range(passes):
        for w in writers:
            w(i)
        got.append(call())
    torch.cuda.synchronize()
    want = []
    for i in range(passes):
        for w in writers:
            w(i)
            torch.cuda.synchronize()
        want.append(call())
        torch.cuda.synchronize()
    return got, want


# the same kernels as above, each behind a launch that writes X and one that writes the bias
@pytest.mark.parametrize("N,K,J", [(512, 512, 20), (512, 2048, 5), (1536, 512, 32), (2048, 512, 100), (32320, 512, 20), (4096, 1024, 500), (2048, 520, 17), (512, 1024, 33)])
@pytest.mark.parametrize("fixed", [False, True])
def test_products_read_what_the_launches_ahead_of_them_wrote(N, K, J, fixed):
    from pimaicompiler_b200 import ops
    ops.init()
    g = torch.Generator(device="cuda").manual_seed(N + K + J)
    W = torch.randn(N, K, generator=g, device="cuda").half() * 0.05
    (X, x_writer), (b, b_writer) = _written(ops, g, (J, K), 12), _written(ops, g, (N,), 12)
    writers = [b_writer, x_writer] if J % 2 else [x_writer, b_writer]
    if not fixed and N * K <= 1 << 20:                          # weights too
        W, w_writer = _written(ops, g, (N, K), 12)
        writers.insert(1, w_writer)
    got, want = _chained(lambda: (ops.gemm_wx_fixed if fixed else ops.gemm_wx)(W, X, b, ops.ACT_RELU), writers, 12)
    assert all(torch.equal(a, w) for a, w in zip(got, want))
    assert len({w.double().sum().item() for w in want}) == 12   # (other operands, other results)


# which operand the launch directly ahead writes, for a matrix times a vector, a vector times a matrix (clusters of several sizes, and
# through memory) and an LSTM cell's step
@pytest.mark.parametrize("form,N,K", [("mv", 1024, 1024), ("mv", 5000, 264), ("mv", 16000, 64), ("vm", 72, 1001), ("vm", 4096, 512), ("vm", 7048, 256), ("vm", 64, 9000)])
@pytest.mark.parametrize("last", ["x", "matrix", "bias"])
def test_vector_products_read_what_the_launches_ahead_of_them_wrote(form, N, K, last):
    from pimaicompiler_b200 import ops
    ops.init()
    g = torch.Generator(device="cuda").manual_seed(N + K)
    made = {"x": _written(ops, g, (K,), 12), "matrix": _written(ops, g, (N, K) if form == "mv" else (K, N), 12), "bias": _written(ops, g, (N,), 12)}
    names = [n for n in made if n != last] + [last]
    m, x, b = made["matrix"][0], made["x"][0], made["bias"][0]
    call = (lambda: ops.gemv_mv(m, x, b)) if form == "mv" else (lambda: ops.gemv_vm(x, m, b))
    got, want = _chained(call, [made[n][1] for n in names], 12)
    assert all(torch.equal(a, w) for a, w in zip(got, want))
    assert len({w.double().sum().item() for w in want}) == 12


@pytest.mark.parametrize("H,I,B", [(320, 320, 12), (512, 1024, 40), (1024, 512, 1), (1024, 512, 70)])
def test_a_cell_reads_what_the_launch_ahead_of_it_wrote(H, I, B):
    from pimaicompiler_b200 import ops
    from tests.util import lstm_params, to_dev
    ops.init()
    g = torch.Generator(device="cuda").manual_seed(H + I)
    m = ops.Lstm([to_dev(p) for p in lstm_params(1, 1, I, H, torch.Generator().manual_seed(H))], 1, False, I, H, True)
    x, writer = _written(ops, g, (B, I), 12)
    h, h_writer = _written(ops, g, (B, H), 12)
    c = torch.randn(1, B, H, generator=g, device="cuda").half()
    got, want = _chained(lambda: torch.cat([t.flatten() for t in m.forward(x.view(1, B, I), h.view(1, B, H), c)]), [h_writer, writer], 12)
    assert all(torch.equal(a, w) for a, w in zip(got, want))
    assert len({w.double().sum().item() for w in want}) == 12
