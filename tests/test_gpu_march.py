"""The 2D march (a warp per strip of 28 columns, rows per warp by the grid's
size) and the step control in an update's last CTA, at the sizes where the
split can go wrong."""
import numpy as np
import pytest

import evora_b200 as ev
from oracle.oracle import Oracle, make_params
from helpers import random_q, rel_l1

pytestmark = pytest.mark.gpu

OPTS = [dict(boundtype=1, limiter=1, solver=2), dict(boundtype=2, limiter=2, solver=1),
        dict(boundtype=3, limiter=3, solver=2), dict(boundtype=3, limiter=1, solver=2),
        dict(boundtype=2, limiter=1, solver=2, secondorder=0)]


def kw_of(nx, ny, opt):
    return dict(nx=nx, ny=ny, nz=1, g=5.0 / 3.0, cfl=0.4, tend=1e9, ymax=ny / nx, **opt)


def state(kw, seed):
    return random_q(Oracle(make_params(**kw)), np.random.default_rng(seed), rho=(0.8, 1.2), vel=(-0.2, 0.2),
                    pres=(0.8, 1.2))


@pytest.mark.parametrize("opt", OPTS, ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()))
@pytest.mark.parametrize("size", [(2, 2), (3, 5), (27, 3), (28, 28), (29, 7), (56, 2), (57, 101), (300, 260)])
def test_march_strict_bitwise(cuda_device, size, opt):
    kw = kw_of(*size, opt)
    q = state(kw, size[0] + size[1])
    want = q.copy()
    r = Oracle(make_params(**kw)).run(want, 6)
    assert r["status"] == 0
    g = ev.Grid(ev.default_params(**kw), ev.FP64, ev.STRICT)
    g.set_q(q)
    g.step(1)          # single steps, and several whose control runs in the updates
    g.step(2)
    g.step(3)
    tm = g.time()
    assert tm["k"] == 6 and tm["t"] == r["t"] and tm["dt"] == r["dt"]
    np.testing.assert_array_equal(g.get_q()[..., :5], want[..., :5])
    g.close()


@pytest.mark.parametrize("precision,flags", [(ev.FP64, 0), (ev.FP32, 0), (ev.FP64, ev.CARRY_ENTROPY),
                                             (ev.FP32, ev.CARRY_ENTROPY)])
@pytest.mark.parametrize("size", [(33, 40), (517, 300), (1500, 900)])
def test_march_forms_match_the_oracle(cuda_device, size, precision, flags):
    """Default FP64 within 1e-12 and FP32 within 1e-5 relative L1 per field
    after 5 steps, as the other kernels' tests have it (the entropy where it
    is carried; else it is derived from the state, not advected)."""
    kw = kw_of(*size, OPTS[0])
    q = state(kw, 5)
    want = q.copy()
    Oracle(make_params(**kw)).run(want, 5)
    g = ev.Grid(ev.default_params(**kw), precision, flags)
    g.set_q(q)
    g.step(5)
    tol = 1e-12 if precision == ev.FP64 else 1e-5
    fields = [0, 1, 2, 4] + ([5] if flags else [])
    assert np.all(rel_l1(g.get_q(), want)[fields] <= tol)
    g.close()


@pytest.mark.parametrize("dims", [(40, 24, 1), (32, 16, 12)])
def test_tail_control_ends_and_stops(cuda_device, dims):
    """The end time falls inside one call; steps after it change nothing.  An
    error raised by a step stops the ones after it."""
    nx, ny, nz = dims
    kw = dict(nx=nx, ny=ny, nz=nz, g=5.0 / 3.0, cfl=0.4, boundtype=2)
    q = state(dict(kw, tend=1e9), 3)
    want = q.copy()
    r = Oracle(make_params(tend=0.02, **kw)).run(want, 1 << 20)
    for stream in (None, "own"):
        import torch
        g = ev.Grid(ev.default_params(tend=0.02, **kw), ev.FP64, ev.STRICT,
                    stream=torch.cuda.Stream() if stream else None)
        g.set_q(q)
        g.step(r["steps"] + 7)
        tm = g.time()
        assert not tm["go"] and tm["k"] == r["steps"] and tm["t"] == r["t"]
        np.testing.assert_array_equal(g.get_q()[..., :5], want[..., :5])
        g.close()
    bad = q.copy()
    bad[nz // 2, ny // 2, nx // 2, 4] = -1.0
    g = ev.Grid(ev.default_params(tend=1.0, **kw))
    g.set_q(bad)
    with pytest.raises(ev.EvoraError):
        g.step(5)
    assert g.status() & 1 and g.time()["k"] == 0
    np.testing.assert_array_equal(g.get_q()[..., :5], bad[..., :5])
    g.close()


@pytest.mark.parametrize("precision,flags", [(ev.FP64, ev.STRICT), (ev.FP32, 0)])
def test_multigrid_kinds_of_members(cuda_device, precision, flags):
    """Batches of 2D members, of 3D members and of both, changed between steps:
    every member equals the grid stepped alone (strict FP64 bit for bit, FP32
    to rounding)."""
    import torch
    stream = torch.cuda.Stream()
    dims = [(57, 33, 1), (300, 70, 1), (24, 20, 18), (2, 2, 1), (33, 9, 40)]
    kws = [dict(nx=a, ny=b, nz=c, g=5.0 / 3.0, cfl=0.4, tend=1e9, boundtype=1 + i % 3, limiter=1 + i % 2,
                solver=2 - i % 2) for i, (a, b, c) in enumerate(dims)]
    qs = [state(kw, i) for i, kw in enumerate(kws)]
    grids = [ev.Grid(ev.default_params(**kw), precision, flags, stream=stream) for kw in kws]
    for g, q in zip(grids, qs):
        g.set_q(q)
    mg = ev.MultiGrid(precision, flags, stream=stream)
    steps = [0] * len(dims)

    def advance(n):
        mg.step(n)
        for i, g in enumerate(grids):
            if g in mg.members:
                steps[i] += n
    for i in (0, 1):
        mg.add(grids[i])
    advance(3)
    for i in (2, 3, 4):
        mg.add(grids[i])
    advance(2)
    for i in (0, 1, 3):
        mg.remove(grids[i])
    advance(3)
    status = mg.status()
    assert [k for _, _, k in status] == [steps[2], steps[4]] and all(e == 0 for _, e, _ in status)
    mg.close()
    for i, (kw, q) in enumerate(zip(kws, qs)):
        with ev.Grid(ev.default_params(**kw), precision, flags) as g:
            g.set_q(q)
            g.step(steps[i])
            if flags:
                np.testing.assert_array_equal(grids[i].get_q(), g.get_q())
            else:
                fields = [0, 1, 2, 4]
                assert np.all(rel_l1(grids[i].get_q(), g.get_q())[fields] <= 1e-5)
        grids[i].close()
