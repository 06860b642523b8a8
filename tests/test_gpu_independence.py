"""A tube's result is the same, bit for bit, in every kernel that may run it:
a cluster of CTAs (few tubes), a CTA per tube (many tubes, or a configured
shape), alone or in a serving mix."""
import numpy as np
import pytest

import evora_b200 as ev
from evora_b200.serving import Server

pytestmark = pytest.mark.gpu

FORMS = {"f32": (ev.FP32, 0, 0), "f32-entropy": (ev.FP32, ev.CARRY_ENTROPY, 0), "f64": (ev.FP64, 0, 0),
         "f64-entropy": (ev.FP64, ev.CARRY_ENTROPY, 0), "f64-dual": (ev.FP64, 0, 1)}
OPTS = [dict(solver=s, limiter=lim, secondorder=so) for s in (1, 2) for lim, so in ((1, 1), (2, 1), (3, 1), (1, 0))]


def opt_id(o):
    return "-".join(f"{k}{v}" for k, v in o.items())


@pytest.mark.parametrize("opt", OPTS, ids=opt_id)
@pytest.mark.parametrize("form", FORMS)
def test_batch_shapes_agree(cuda_device, form, opt):
    precision, flags, dual = FORMS[form]
    for bt in (1, 2, 3):
        kw = dict(g=5.0 / 3.0, cfl=0.6, boundtype=bt, dualenergy=dual, tend=0.01, **opt)
        lengths, q = ev.ic.random_tubes(12, seed=5, nmin=40, nmax=900)
        p = ev.default_params(nx=max(lengths), ny=1, nz=1, **kw)
        first = None
        for threads in (None, 128, 256, 512):      # None: the default, a cluster per tube
            with ev.Batch(p, lengths, precision, flags) as b:
                if threads:
                    b.configure(threads, 1)
                b.set_q(q)
                b.run()
                got = b.get_q(), [b.info(i) for i in range(len(lengths))]
            first = first or got
            assert got[1] == first[1]
            np.testing.assert_array_equal(got[0], first[0])


@pytest.mark.parametrize("solver", [1, 2])
@pytest.mark.parametrize("form", ["f32", "f32-entropy", "f64"])
def test_serving_alone_equals_mix(cuda_device, form, solver):
    """170 tubes in flight take a CTA each, a few of them a cluster each."""
    precision, flags, _ = FORMS[form]
    lengths, q = ev.ic.random_tubes(170, seed=9, nmin=40, nmax=500)
    offs = np.concatenate([[0], np.cumsum(lengths)])

    def serve(which):
        p = ev.default_params(g=5.0 / 3.0, cfl=0.6, boundtype=1, solver=solver, limiter=1)
        with Server(p, precision, flags, steps_per_tick=16, max_tube_cells=1024, max_tubes=256) as s:
            ids = [s.submit(np.ascontiguousarray(q[offs[i]:offs[i + 1]]), 0.005) for i in which]
            while s.tick() != (0, 0):
                pass
            return [s.result(i) for i in ids]

    mix = serve(range(170))
    for i in (0, 77, 169):
        alone = serve([i])[0]
        assert alone[2:] == mix[i][2:]
        np.testing.assert_array_equal(alone[0], mix[i][0])
