"""The limiters of the fast forms on differences whose product leaves the
range of the type."""
import numpy as np
import pytest

import evora_b200 as ev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,small,tol", [(ev.FP32, 2.0 ** -70, 1e-5), (ev.FP64, 2.0 ** -600, 1e-12)])
@pytest.mark.parametrize("dims", [(200, 1, 1), (48, 40, 1), (24, 20, 18)])
def test_moncen_small_differences(cuda_device, dims, precision, small, tol):
    """A transverse velocity far below the sound speed is carried along
    passively, so its momentum scales with its amplitude: by a power of two,
    to rounding.  The monotonised central limiter compares signs
    (muscl.f90:141-154), so its slopes do not vanish where the product of two
    differences underflows.  The other run's amplitude is small enough for its
    kinetic energy to be lost in the rounding of E."""
    nx, ny, nz = dims
    kw = dict(nx=nx, ny=ny, nz=nz, g=5.0 / 3.0, cfl=0.4, boundtype=2, solver=2, limiter=2, tend=1e9)
    x = np.broadcast_to(2 * np.pi * (np.arange(nx) + 0.5) / nx, (nz, ny, nx))
    rho, v = 1.0 + 0.3 * np.sin(x), 0.2 * np.cos(x)
    got = []
    for a in (small, 2.0 ** -16 if precision == ev.FP32 else 2.0 ** -40):
        q = np.zeros((nz, ny, nx, 6))
        q[..., 0], q[..., 1], q[..., 3] = rho, rho * v, a * rho * np.sin(2 * x)
        q[..., 4] = 0.5 * rho * v * v + 1.5
        q[..., 5] = 1.0 / rho ** (2.0 / 3.0)
        with ev.Grid(ev.default_params(**kw), precision) as g:
            g.set_q(q)
            g.step(10)
            got.append(g.get_q()[..., 3] / a)
    assert np.abs(got[0] - got[1]).sum() <= tol * np.abs(got[1]).sum()
