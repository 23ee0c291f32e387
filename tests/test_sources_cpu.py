"""CPU: rules that the CUDA sources keep and no compiler checks."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pimaicompiler_b200", "csrc")


def _kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\(", text):
        start = text.index("{", m.end())
        depth, i = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.start():start], text[start:i]


def test_kernels_that_wait_for_their_predecessor_read_its_outputs_by_plain_loads():
    # a launch that starts early may overlap the kernel that writes its inputs: nothing behind the wait goes through the
    # read-only path, but constants of a handle (said beside them)
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for name, parameters, body in _kernels(open(path).read()):
            if "pdl_wait();" not in body:
                continue
            seen += 1
            where = f"{os.path.basename(path)}: {name}"
            assert not re.search(r"const [^,]*__restrict__", parameters), where + ": a read-only parameter"
            for line in body[body.index("pdl_wait();"):].splitlines():
                assert not re.search(r"__ldg\(|\bldg_|global\.nc", line) or "constant of the handle" in line, where + ": " + line.strip()
    assert seen >= 15


def test_loads_behind_a_wait_are_volatile():
    text = "".join(open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))))
    loads = re.findall(r"(asm\b[^;]{0,12}\(\s*\"ld\.global[^\"]*)", text)
    assert loads and all("volatile" in a for a in loads if ".nc" not in a)
