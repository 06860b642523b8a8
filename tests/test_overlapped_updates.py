"""2D updates launched while the previous one still runs (programmatic
dependent launch) read a state that is being written."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evora_b200", "csrc")


def test_march_reads_its_state_coherently():
    """The non-coherent load path (ld(), __ldg, const __restrict__) is for
    data that does not change in the kernel's lifetime, which here begins
    before the previous update's stores."""
    with open(os.path.join(CSRC, "fused_march.cuh")) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert "step_head();" in code
    assert not re.search(r"\bld\(|__ldg|__restrict__|ld\.global\.nc", code)


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(24, 20), (64, 64), (333, 250)])
def test_overlapped_updates_equal_separate_ones(cuda_device, size):
    """Event timing launches the updates one after the other: 400 steps both
    ways, strict FP64 bit for bit."""
    import evora_b200 as ev
    import torch
    nx, ny = size
    p = ev.default_params(nx=nx, ny=ny, nz=1, g=5.0 / 3.0, cfl=0.4, boundtype=2, tend=1e9)
    q = ev.ic.kh2d(p)
    got = []
    for timed in (False, True):
        g = ev.Grid(p, ev.FP64, ev.STRICT, stream=torch.cuda.Stream())
        g.set_timing(timed)
        g.set_q(q)
        g.step(400)
        got.append((g.get_q(), g.time()))
        g.close()
    assert got[0][1] == got[1][1] and got[0][1]["k"] == 400
    np.testing.assert_array_equal(got[0][0], got[1][0])
