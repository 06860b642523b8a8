"""The launches that a member of a multi-grid batch reports."""
import pytest

import evora_b200 as ev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,chunks", [(1, 1), (32, 1), (33, 2), (70, 3)])
def test_multigrid_launches(cuda_device, steps, chunks):
    """Per step a control kernel and an update per kind of members, and a
    closing control kernel per graph of at most 32 steps."""
    import torch
    stream = torch.cuda.Stream()
    grids = []
    with ev.MultiGrid(ev.FP32, stream=stream) as mg:
        for n, nz in ((16, 1), (24, 12)):
            p = ev.default_params(nx=n, ny=n, nz=nz, g=5.0 / 3.0, cfl=0.4, boundtype=2, tend=1e9)
            grids.append(ev.Grid(p, ev.FP32, stream=stream))
            grids[-1].set_q(ev.ic.kh2d(p) if nz == 1 else ev.ic.kh3d(p, seed=1))
            grids[-1].set_timing(True)
            mg.add(grids[-1])
        mg.step(steps)
        for g in grids:
            assert g.timing()["launches"] == 3 * steps + chunks
            assert g.time()["k"] == steps
    for g in grids:
        g.close()
