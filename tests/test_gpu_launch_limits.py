"""Batches, servers and 1D grids of different lengths share kernels, whose
limit of dynamic shared memory is one per kernel: none may lower it under
another."""
import threading

import numpy as np
import pytest

import evora_b200 as ev
from evora_b200.serving import Server

pytestmark = pytest.mark.gpu

KW = dict(g=5.0 / 3.0, cfl=0.4, boundtype=2, solver=2, limiter=1, tend=1e9)


def tubes(n, count):
    return ev.ic.random_tubes(count, seed=n, nmin=n, nmax=n)


def advance(b):
    assert b.run(max_steps=3) == 0
    assert all(b.info(i)["k"] == 3 for i in range(len(b.n)))
    return b.get_q()


@pytest.mark.parametrize("precision", [ev.FP64, ev.FP32])
@pytest.mark.parametrize("long,short,count", [(2500, 1000, 200), (900, 500, 700), (8000, 3000, 5)])
def test_a_shorter_batch_leaves_a_longer_one_alone(cuda_device, long, short, count, precision):
    """One kernel and shape for both: a CTA per tube, and a cluster per tube."""
    first = {}
    for lives in (1, 2):
        made = []
        for n in (long, short)[:lives] if lives == 2 else (long,):
            lengths, q = tubes(n, count)
            made.append(ev.Batch(ev.default_params(nx=n, ny=1, nz=1, **KW), lengths, precision))
            made[-1].set_q(q)
        if lives == 2:
            advance(made[1])
        first[lives] = advance(made[0])
        for b in made:
            b.close()
    np.testing.assert_array_equal(first[1], first[2])


def test_a_batch_leaves_a_server_alone(cuda_device):
    """The server's kernel and the batch's are the same (768 threads); 160
    requests, admitted over two rounds, take a CTA per tube."""
    lengths, q = tubes(3000, 160)
    reqs = q.reshape(160, 3000, 6)
    base = ev.default_params(g=KW["g"], cfl=KW["cfl"], boundtype=2, solver=2, limiter=1)
    with Server(base, ev.FP32, steps_per_tick=1, max_tube_cells=5600, max_tubes=256) as s:
        ids = [s.submit(np.ascontiguousarray(r), 1e-3) for r in reqs]
        with ev.Batch(ev.default_params(nx=3000, ny=1, nz=1, **KW), lengths, ev.FP32) as b:
            b.set_q(q)
            advance(b)
            while s.tick() != (0, 0):
                pass
        assert all(s.result(i)[3] == 0 for i in ids)


def test_two_threads_with_lines_of_different_length(cuda_device):
    import torch
    done = {}

    def work(n):
        lengths, q = tubes(n, 1)
        g = ev.Grid(ev.default_params(nx=n, ny=1, nz=1, **KW), ev.FP64, stream=torch.cuda.Stream())
        g.set_q(q.reshape(1, 1, n, 6))
        for _ in range(1500):
            g.step(1, sync=False)
        g.step(1)
        done[n] = g.time()["k"]
        g.close()

    threads = [threading.Thread(target=work, args=(n,)) for n in (7900, 1000, 5000, 300)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert done == {7900: 1501, 1000: 1501, 5000: 1501, 300: 1501}
