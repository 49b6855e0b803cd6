"""Device initial conditions keep a column's z-independent factors and take a
chunk of planes per thread: perturbed and unperturbed lines along every axis,
products in both orders, grids of one plane per thread and of several, against
the host's formulas; and multiply_ic over the same columns."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200 import ic
from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def params(shape, storage="c128"):
    nx, ny, nz = shape
    return RunParams(nx=nx, ny=ny, nz=nz, xr=0.2 * (nx - 1), yr=0.21 * (ny - 1), zr=0.19 * (nz - 1), mu=2.0, omx=0.1,
                     omy=0.2, omz=0.15, bcs=2, order=4, storage=storage)


def host(rp, names, line, ring):
    out = None
    for n in names:
        v = {"fermi": lambda: ic.fermi(rp), "line": lambda: ic.vortex_line(rp, **line),
             "line_pade": lambda: ic.vortex_line_pade(rp, **line), "ring": lambda: ic.vortex_ring(rp, "yz", **ring),
             "vortex_pair": lambda: ic.vortex_pair(rp), "sphere": lambda: ic.sphere(rp)}[n]()
        out = v if out is None else out * v
    return out


LINES = [dict(x0=0.3, y0=-0.2, dir="z"), dict(y0=0.1, z0=0.4, dir="x", sgn=-1.0), dict(x0=-0.2, dir="y"),
         dict(x0=0.1, dir="z", amp1=0.3, amp2=0.2, ll=3.0), dict(dir="z", sgn=2.0)]


@pytest.mark.parametrize("shape", [(6, 7, 9), (33, 9, 40), (96, 200, 70)])
@pytest.mark.parametrize("line", range(len(LINES)))
@pytest.mark.parametrize("names", [("fermi", "line_pade"), ("line", "fermi", "vortex_pair"), ("ring", "line")])
def test_products_over_columns(gpu, shape, line, names):
    rp = params(shape)
    ring = dict(r0=1.0) if line % 2 else dict(r0=1.0, amp=0.1, mm=2, r1=0.05, kk=3)
    kw = dict(ring=dict(plane="yz", **ring), line=LINES[line])
    s = Solver(rp)
    s.set_ic(ic.device_spec(*names, **kw))
    ref = host(rp, names, LINES[line], ring)
    tol = 1e-13 * max(1.0, float(np.abs(ref).max()))
    # a perturbed ring depends on the angle about its axis (y = z = 0), which
    # has no value on it: the oracle has none there either
    _, y, z, _ = s.grid()
    defined = (np.hypot(y[None, :, None], z[:, None, None]) > 1e-12) | ("ring" not in names) | ("amp" not in ring)
    ref = np.where(defined, ref, s.get_state())
    np.testing.assert_allclose(s.get_state(), ref, rtol=0, atol=tol)
    s.multiply_ic(ic.device_spec("line_pade", **kw), modulus=True)
    np.testing.assert_allclose(s.get_state(), np.abs(ref) * host(rp, ("line_pade",), LINES[line], ring), rtol=0,
                               atol=4 * tol * float(np.abs(ref).max() + 1))
    # the ghosts the kernel wrote are those of a packed state
    e = s.energy()
    t = Solver(rp)
    t.set_state(s.get_state())
    assert t.energy() == e
    s.close()
    t.close()
