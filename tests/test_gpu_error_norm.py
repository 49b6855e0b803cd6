"""The RKF45 error norm: the march passes over sites whose ratio cannot exceed
the largest so far.  Its maximum equals that of the kernel which evaluates
every site, whatever the scale of the state (the screen works in single
precision), with zeros in it and in imaginary time."""
from __future__ import annotations

import os

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def run(rp, psi, march):
    # 40 x 21 x 26 is a small grid: one thread per site unless a chunk is asked for
    old = os.environ.pop("GPE_ZC", None)
    if march:
        os.environ["GPE_ZC"] = str(march)
    try:
        s = Solver(rp)
    finally:
        os.environ.pop("GPE_ZC", None)
        if old is not None:
            os.environ["GPE_ZC"] = old
    s.set_state(psi)
    out = [(i.errmax, i.rejected, s.dt) for i in (s.solver(1) for _ in range(3))]
    state = s.get_state()
    s.close()
    return out, state


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-25, 1e-160, 1e12, 1e25, 1e150])
@pytest.mark.parametrize("real_time", [True, False])
@pytest.mark.parametrize("zeros", [False, True])
def test_error_norm_equals_every_site(gpu, scale, real_time, zeros):
    # g = 0: the step is linear, so the ratio does not depend on the scale
    rp = RunParams(nx=40, ny=21, nz=26, xr=4.875, yr=2.5, zr=3.125, tau=1e-3, scheme="rk45", eqn_to_solve=4, bcs=2,
                   order=4, g=0.0, mu=1.0, omx=0.3, omy=0.2, gamma=0.05, real_time=real_time)
    rng = np.random.default_rng(3)
    psi = scale * (1.0 + 0.1 * (rng.normal(size=(26, 21, 40)) + 1j * rng.normal(size=(26, 21, 40))))
    if zeros:
        psi[5:20, 4:16, 6:30] = 0.0
    ref, sref = run(rp, psi, 0)
    for march in (26, 7):
        out, state = run(rp, psi, march)
        assert out == ref
        np.testing.assert_array_equal(state, sref)


def test_error_norm_complex64(gpu):
    rp = RunParams(nx=40, ny=21, nz=26, xr=4.875, yr=2.5, zr=3.125, tau=1e-3, scheme="rk45", eqn_to_solve=4, bcs=1,
                   order=2, g=1.0, mu=1.0, storage="c64")
    rng = np.random.default_rng(4)
    psi = 1.0 + 0.1 * (rng.normal(size=(26, 21, 40)) + 1j * rng.normal(size=(26, 21, 40)))
    ref, sref = run(rp, psi, 0)
    out, state = run(rp, psi, 7)
    assert out == ref
    np.testing.assert_array_equal(state, sref)
