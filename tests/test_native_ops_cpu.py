"""CPU: the native call path of the short ops with arguments that never reach the device."""
import subprocess
import sys

CODE = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from pimaicompiler_b200 import _lib

def fake(*shape):
    with FakeTensorMode():
        return torch.empty(*shape, dtype=torch.half, device="cuda")

ops = _lib.native()
for call in (lambda: ops.gemv_mv(fake(16, 8), fake(8), None, 0, fake(16)),
             lambda: ops.gemv_vm(fake(8), fake(8, 16), None, 0, fake(16)),
             lambda: ops.gemm_wx(fake(16, 8), fake(4, 8), None, 0, False, fake(4, 16)),
             lambda: ops.gemm_wx(fake(16, 8), fake(4, 8), None, 0, False, fake(())),
             lambda: ops.lstm_forward(0, 1, 1, 16, fake(5, 2, 8), None, None, False, (fake(5, 2, 16), fake(1, 2, 16), fake(1, 2, 16)))):
    try:
        call()
    except Exception:
        continue
    raise SystemExit("not refused")
"""


def test_tensors_without_memory_are_refused_with_an_exception():
    # a tracer's tensors have no address; asking for one inside the call of the C ABI ended the process
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])
