"""The library's work is ordered on its own non-blocking streams alone.  A
non-blocking stream does not wait for the legacy default stream, so a memset or
copy issued there could land after the kernels that rely on it."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bonsai2_b200", "csrc")


def test_no_default_stream_operation_in_the_sources():
    """Every memset, copy and launch names its stream.  (The symbol copies of
    bounds-checked builds are the host's own reads of a counter, after a
    synchronize.)"""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"\bcudaMem(?:set|cpy)(?:2D|3D)?\s*\(", src):
            found.append((os.path.basename(path), m.group(0)))
        for m in re.finditer(r"<<<(.*?)>>>", src, flags=re.S):
            depth, args = 0, 1
            for ch in m.group(1):
                depth += ch in "([{"
                depth -= ch in ")]}"
                args += ch == "," and depth == 0
            if args != 4:
                found.append((os.path.basename(path), m.group(0)))
    assert not found, found


@pytest.mark.gpu
@pytest.mark.parametrize("systems", [None, (3000, 1, 5000)])
def test_handles_made_while_the_default_stream_is_busy(lib, systems):
    """Handles created, allocated, loaded and stepped with work of another
    library queued on the default stream give what they give without it."""
    import torch

    import bonsai2_b200 as B
    n = 9000 if systems is None else sum(systems)
    pos, vel = B.plummer(n, 8)
    a = torch.randn(4096, 4096, device="cuda")

    def run(busy):
        torch.cuda.synchronize()
        if busy:
            b = a
            for _ in range(20):  # some tens of milliseconds
                b = torch.tanh(b @ a)
        t = B.Treecode(eps=0.01, theta=0.6)
        t.set_precision(1)
        if systems is None:
            t.alloc(n)
        else:
            t.set_systems(np.array(systems, np.int32))
        t.set_block_steps(1, 0.2)
        t.h_ptclPos[:] = pos
        t.h_ptclVel[:] = vel
        t.ptcl_h2d()
        t.step(2)
        t.block_step(1)
        status = t.synchronize()
        torch.cuda.synchronize()
        t.ptcl_d2h()
        out = t.h_ptclPos.copy(), t.h_ptclVel.copy(), t.get_acc(), t.levels()
        t.close()
        assert status == 0
        return out

    quiet = run(False)
    for _ in range(3):
        for x, y in zip(quiet, run(True)):
            assert np.array_equal(x, y)
