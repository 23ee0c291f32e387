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
