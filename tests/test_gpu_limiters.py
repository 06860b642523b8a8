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


@pytest.mark.parametrize("precision", [ev.FP32, ev.FP64])
@pytest.mark.parametrize("limiter", [2, 3])
@pytest.mark.parametrize("dims", [(300, 1, 1), (60, 50, 1), (22, 20, 18)])
def test_nan_cell_raises_the_literal_forms_errors(cuda_device, dims, limiter, precision):
    """A NaN in one cell: the slopes beside it are those of the literal forms
    (strict FP64) as far as the raised errors tell, with HLL and with HLLC."""
    nx, ny, nz = dims
    rng = np.random.default_rng(1)
    sh = dims[::-1]
    rho, v, p = rng.uniform(0.5, 2, sh), rng.uniform(-0.5, 0.5, sh + (3,)), rng.uniform(0.5, 2, sh)
    v[..., 1] *= ny > 1
    v[..., 2] *= nz > 1
    q = np.empty(sh + (6,))
    q[..., 0], q[..., 1:4] = rho, rho[..., None] * v
    q[..., 4], q[..., 5] = 0.5 * rho * (v * v).sum(-1) + 1.5 * p, p / rho ** (2.0 / 3.0)
    q.reshape(-1, 6)[7, 1] = np.nan
    for solver, bt in ((1, 3), (2, 2)):
        kw = dict(nx=nx, ny=ny, nz=nz, g=5.0 / 3.0, cfl=0.3, boundtype=bt, solver=solver, limiter=limiter, tend=1e9)
        status = []
        for prec, flags in ((ev.FP64, ev.STRICT), (precision, 0)):
            with ev.Grid(ev.default_params(**kw), prec, flags) as g:
                g.set_q(q)
                with pytest.raises(ev.EvoraError):
                    g.step(4)
                status.append(g.status())
        assert status[0] == status[1]
