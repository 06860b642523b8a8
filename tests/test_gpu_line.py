"""1D grids whose steps run inside one cluster launch (k_steps1d) and tubes
whose cells are updated in chunks of 30 per warp (tube_sweep), at the sizes
where the split can go wrong: single chunks and ranks, their remainders, the
changes of the number of ranks, both ends of the range."""
import numpy as np
import pytest

import evora_b200 as ev
from oracle.oracle import Oracle, make_params
from helpers import random_q, rel_l1

pytestmark = pytest.mark.gpu

OPTS = [dict(boundtype=1, limiter=1, solver=2), dict(boundtype=2, limiter=2, solver=1),
        dict(boundtype=3, limiter=3, solver=2), dict(boundtype=2, limiter=1, solver=2, secondorder=0)]


def kw_of(n, opt):
    return dict(nx=n, ny=1, nz=1, g=5.0 / 3.0, cfl=0.4, tend=1e9, **opt)


# 1 rank up to 96 cells, 2 to 300, 4 to 700, 8 to 8000 (FP64), 16 above
@pytest.mark.parametrize("opt", OPTS, ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()))
@pytest.mark.parametrize("n", [2, 3, 30, 31, 96, 97, 300, 301, 700, 702, 1024, 1929, 8000, 8001])
def test_steps1d_strict_bitwise(cuda_device, n, opt):
    o = Oracle(make_params(**kw_of(n, opt)))
    q = random_q(o, np.random.default_rng(n))
    want = q.copy()
    steps = 9
    o.run(want, steps)
    g = ev.Grid(ev.default_params(**kw_of(n, opt)), ev.FP64, ev.STRICT)
    g.set_q(q)
    g.step(2)
    g.step(steps - 2)
    got = g.get_q()
    tm = g.time()
    g.close()
    assert tm["k"] == steps and tm["go"]
    assert np.array_equal(got[..., :5], want[..., :5])


@pytest.mark.parametrize("nf6", [0, ev.CARRY_ENTROPY])
@pytest.mark.parametrize("precision", [ev.FP64, ev.FP32])
@pytest.mark.parametrize("n", [2, 97, 701, 1024, 11000])
def test_steps1d_matches_separate_kernels(cuda_device, n, precision, nf6):
    """Event timing keeps a kernel per part of the step: the same run both
    ways.  The arithmetic of a cell is the same, up to the contraction of its
    products: FP64 to 1e-13, FP32 to 1e-5 relative L1 after 20 steps."""
    p = ev.default_params(**kw_of(n, OPTS[0]))
    q = random_q(Oracle(make_params(**kw_of(n, OPTS[0]))), np.random.default_rng(n + 1))
    res = []
    for timed in (False, True):
        g = ev.Grid(p, precision, nf6)
        g.set_timing(timed)
        g.set_q(q)
        g.step(20)
        res.append((g.get_q(), g.time()))
        g.close()
    tol = 1e-13 if precision == ev.FP64 else 1e-5
    assert np.all(rel_l1(res[0][0], res[1][0])[[0, 1, 4, 5]] <= tol)
    assert res[0][1]["k"] == res[1][1]["k"] == 20
    assert abs(res[0][1]["t"] - res[1][1]["t"]) <= 20 * tol * res[1][1]["t"]


def test_steps1d_end_and_error(cuda_device):
    """The end time stops the run inside a launch; a cell without pressure
    stops it before its update, with the state and the step count kept."""
    kw = dict(kw_of(1000, OPTS[0]), tend=0.01)
    o = Oracle(make_params(**kw))
    q = random_q(o, np.random.default_rng(8))
    want = q.copy()
    o.run(want, 1 << 20)
    g = ev.Grid(ev.default_params(**kw), ev.FP64, ev.STRICT)
    g.set_q(q)
    g.step(5000)
    tm = g.time()
    assert not tm["go"] and tm["t"] == 0.01
    assert np.array_equal(g.get_q()[..., :5], want[..., :5])
    bad = q.copy()
    bad[0, 0, 777, 4] = 0.0
    g.set_q(bad)
    with pytest.raises(ev.EvoraError):
        g.step(5)
    assert g.status() == 1 and g.time()["k"] == 0
    assert np.array_equal(g.get_q()[..., :5], bad[..., :5])
    g.close()


@pytest.mark.parametrize("lengths", [[2, 3, 29, 30, 31, 59, 60, 61, 119, 121], [480, 481, 510, 512, 961],
                                     [1500] * 300 + [31, 2], [3000] * 3])
def test_tubes_strict_bitwise_at_chunk_edges(cuda_device, lengths):
    """Every default CTA shape, at lengths around whole chunks."""
    kw = dict(g=5.0 / 3.0, cfl=0.4, boundtype=3, limiter=2, solver=2, tend=1e9)
    rng = np.random.default_rng(len(lengths))
    qs, want = [], []
    for i, n in enumerate(lengths):
        o = Oracle(make_params(nx=n, ny=1, nz=1, **kw))
        q = random_q(o, rng) if i < 10 or n < 100 else qs[i % 10].copy()
        qs.append(q)
        w = q.copy()
        if i < 10 or n < 100:
            o.run(w, 7)
        want.append(w if i < 10 or n < 100 else want[i % 10])
    b = ev.Batch(ev.default_params(nx=max(lengths), ny=1, nz=1, **kw), lengths, ev.FP64, ev.STRICT)
    b.set_q(np.concatenate([q.reshape(-1, 6) for q in qs]))
    assert b.run(max_steps=7) == 0
    got = b.get_q()
    b.close()
    ref = np.concatenate([w.reshape(-1, 6) for w in want])
    assert np.array_equal(got[:, :5], ref[:, :5])


@pytest.mark.parametrize("bt", [1, 2, 3])
@pytest.mark.parametrize("lengths", [[2, 63, 64, 65, 66, 127, 129], [511, 512, 513, 1025] * 9, [2049, 3000, 8] * 40,
                                     [5000, 14000]])
def test_tube_clusters_strict_bitwise(cuda_device, lengths, bt):
    """Small batches (clusters of 8, 4 and 2 CTAs per tube, and one CTA for the
    lengths that fit none) against the configured shape and the oracle."""
    kw = dict(g=5.0 / 3.0, cfl=0.4, boundtype=bt, limiter=1, solver=2, tend=1e9)
    rng = np.random.default_rng(len(lengths))
    states = {}
    for n in set(lengths):
        o = Oracle(make_params(nx=n, ny=1, nz=1, **kw))
        q = random_q(o, rng)
        w = q.copy()
        o.run(w, 5)
        states[n] = (q.reshape(-1, 6), w.reshape(-1, 6))
    q = np.concatenate([states[n][0] for n in lengths])
    for configured in (False, True):
        b = ev.Batch(ev.default_params(nx=max(lengths), ny=1, nz=1, **kw), lengths, ev.FP64, ev.STRICT)
        if configured:
            b.configure(256, 1)
        b.set_q(q)
        assert b.run(max_steps=2) == 0 and b.run(max_steps=3) == 0
        got = b.get_q()
        assert all(b.info(i)["k"] == 5 for i in range(0, len(lengths), 7))
        b.close()
        assert np.array_equal(got[:, :5], np.concatenate([states[n][1] for n in lengths])[:, :5])


def test_tube_clusters_end_and_error(cuda_device):
    """Tubes of a small batch end at their own times and fail alone."""
    lengths, q = ev.ic.random_tubes(12, seed=4, nmin=100, nmax=900)
    p = ev.default_params(nx=max(lengths), ny=1, nz=1, g=5.0 / 3.0, cfl=0.8, boundtype=1, solver=2, tend=0.02)
    offs = np.concatenate([[0], np.cumsum(lengths)])
    q[offs[3] + 5, 4] = -1.0
    res = []
    for configured in (False, True):
        b = ev.Batch(p, lengths, ev.FP64, ev.STRICT)
        if configured:
            b.configure(256, 1)
        b.set_tend(2, 0.01)
        b.set_q(q)
        b.run()
        res.append((b.get_q(), [b.info(i) for i in range(12)]))
        b.close()
    assert res[0][1] == res[1][1]
    assert res[0][1][3]["status"] == 2 and res[0][1][3]["k"] == 0 and res[0][1][3]["err"] & 1
    assert res[0][1][2]["t"] == 0.01 and all(i["status"] == 1 for j, i in enumerate(res[0][1]) if j != 3)
    assert np.array_equal(res[0][0], res[1][0])
