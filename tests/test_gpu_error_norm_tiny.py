"""RKF45 error norms so small that their squares leave the range of normal
floats, on states so large that the squared scale does not: the march's
single-precision screen may pass over no site that holds the largest ratio."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def run(rp, psi):
    with Solver(rp) as s:
        s.set_state(psi)
        out = [(i.errmax, i.rejected, s.dt) for i in (s.solver(1) for _ in range(3))]
        return out, s.get_state()


# The first step's largest ratio is rounding error, about 1.6e-15 tau here; a
# time step grows five times from step to step.  All ratios from 2.65e-23 to
# 3.74e-23 have the same square in floats, the smallest there is.
@pytest.mark.parametrize("tau", [1e-8, 1.8e-8, 2e-8, 2.1e-8, 2.2e-8, 2.3e-8, 2.8e-8, 1e-7, 1e-5])
@pytest.mark.parametrize("scale", [1e5, 1e9])
def test_error_norm_equals_every_site(gpu, tau, scale):
    # one thread per site looks at every site; chunks of planes screen all but their first
    rp = RunParams(nx=40, ny=21, nz=26, xr=4.875, yr=2.5, zr=3.125, tau=tau, scheme="rk45", eqn_to_solve=4, bcs=2,
                   order=4, g=0.0, mu=1.0, omx=0.3, omy=0.2)
    rng = np.random.default_rng(8)
    psi = scale * (1.0 + 0.1 * (rng.normal(size=(26, 21, 40)) + 1j * rng.normal(size=(26, 21, 40))))
    ref, sref = run(rp, psi)
    for march in (26, 7):
        out, state = run(rp.replace(tile_zc=march), psi)
        assert out == ref
        np.testing.assert_array_equal(state, sref)


# a trapped state with nothing, next to nothing and less than the scale's own
# 1e-30 around it; attempts that are rejected until dt is far below the one at entry
@pytest.mark.parametrize("outside", [0.0, 1e-12, 1e-20, 1e-31, 1e-80, 1e-170])
@pytest.mark.parametrize("storage", ["c128", "c64"])
@pytest.mark.parametrize("real_time,tau", [(True, 1e-3), (False, 1e-3), (True, 0.2)])
def test_vacuum(gpu, outside, storage, real_time, tau):
    if outside and storage == "c64" and outside < 1e-30:
        outside = 1e-38  # (the storage's own smallest)
    rp = RunParams(nx=40, ny=21, nz=26, xr=4.875, yr=2.5, zr=3.125, tau=tau, scheme="rk45", eqn_to_solve=4, bcs=2,
                   order=4, g=1.0, mu=1.0, omx=0.3, omy=0.2, gamma=0.05 if real_time else 0.0, real_time=real_time,
                   storage=storage)
    rng = np.random.default_rng(9)
    psi = 1.0 + 0.1 * (rng.normal(size=(26, 21, 40)) + 1j * rng.normal(size=(26, 21, 40)))
    full = np.zeros(psi.shape, bool)
    full[6:18, 5:14, 8:20] = True
    psi = np.where(full, psi, outside * psi)
    ref, sref = run(rp, psi)
    for march in (26, 7):
        out, state = run(rp.replace(tile_zc=march), psi)
        assert out == ref
        np.testing.assert_array_equal(state, sref)
