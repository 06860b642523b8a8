"""The CTA shapes of batched tubes: the default one without tuning, the tuned
one, and explicit ones."""
import numpy as np
import pytest

import evora_b200 as ev

pytestmark = pytest.mark.gpu


def ms(lengths, q, precision, prepare=None):
    import torch
    p = ev.default_params(nx=max(lengths), ny=1, nz=1, g=5.0 / 3.0, cfl=0.4, boundtype=2, tend=1e9)
    stream = torch.cuda.Stream()
    with ev.Batch(p, lengths, precision) as b:
        b.set_stream(stream)
        b.set_q(q)
        if prepare:
            prepare(b)
        b.run(max_steps=20)
        times = []
        for _ in range(5):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record(stream)
            b.run(max_steps=20, sync=False)
            e1.record(stream)
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
    return min(times)


# 15 %: what neighbouring shapes differ by at a change of the rule
@pytest.mark.parametrize("n,precision", [(3000, ev.FP32), (4096, ev.FP32), (3000, ev.FP64)])
def test_default_shape_of_many_long_tubes(cuda_device, n, precision):
    lengths, q = ev.ic.random_tubes(600, seed=n, nmin=n, nmax=n)
    assert ms(lengths, q, precision) <= 1.15 * ms(lengths, q, precision, lambda b: b.configure(512, 1))


def test_tuned_small_batch_is_no_slower(cuda_device):
    """The tuner knows the clusters that a small batch runs in by default."""
    lengths, q = ev.ic.random_tubes(20, seed=2, nmin=3000, nmax=3000)
    tuned = ms(lengths, q, ev.FP32, lambda b: b.autotune(steps=20))
    assert tuned <= 1.15 * ms(lengths, q, ev.FP32)


def test_explicit_and_reported_shapes(cuda_device):
    """768 threads are a shape of its own, with 5 fields; the tuner reports the
    shape that it leaves, and it can be set again."""
    lengths, q = ev.ic.random_tubes(300, seed=3, nmin=2900, nmax=3100)
    p = ev.default_params(nx=max(lengths), ny=1, nz=1, g=5.0 / 3.0, cfl=0.4, boundtype=2, tend=1e9)
    got = []
    with ev.Batch(p, lengths, ev.FP32) as b:
        for shape in (None, (512, 1), (768, 1), "tuned", "again"):
            if shape == "tuned":
                tuned = b.autotune(steps=3)
                assert tuned[0] in (128, 256, 512, 768) and tuned[1] in (1, 2, 3)
            elif shape:
                b.configure(*(tuned if shape == "again" else shape))
            b.set_q(q)
            assert b.run(max_steps=4) == 0
            got.append(b.get_q())
        for bad in ((64, 1), (1024, 1), (768, 0), (768, 9)):
            with pytest.raises(ev.EvoraError):
                b.configure(*bad)
    for other in got[1:]:
        np.testing.assert_array_equal(other, got[0])
    with ev.Batch(p, lengths[:3], ev.FP32, ev.CARRY_ENTROPY) as b:
        with pytest.raises(ev.EvoraError):
            b.configure(768, 1)
