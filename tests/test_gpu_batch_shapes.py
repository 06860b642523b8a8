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
