"""Axes so long that a launch's limit of 65535 blocks along y and z bounds the
shape of the initial-state and stage launches: they are accepted and right."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200 import ic
from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


# order 2 along z would like 16 planes a CTA; 16-row tiles along y
@pytest.mark.parametrize("shape,storage,order", [((6, 6, 1100000), "c128", 2), ((6, 600000, 6), "c64", 4)])
def test_long_axes(gpu, shape, storage, order):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.001,
                   scheme="euler", eqn_to_solve=4, bcs=2, order=order, g=2.0, mu=1.0, storage=storage)
    with Solver(rp) as s:
        s.set_ic(ic.device_spec("wall"))  # 0 for z <= -30, else 1
        _, _, z, _ = s.grid()
        psi = np.broadcast_to(np.where(z <= -30.0, 0.0, 1.0)[:, None, None], (nz, ny, nx))
        np.testing.assert_array_equal(s.get_state(), psi)
        s.set_ic(ic.device_spec("uniform"))
        s.solver(1)
        # psi' = psi - i dt (g |psi|^2 psi - mu psi) at every site of a uniform state
        out = s.get_state()
        want = complex(1.0, -0.001)
        assert np.abs(out - want).max() <= (4e-16 if storage == "c128" else 2.0 ** -24)
