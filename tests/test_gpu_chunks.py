"""The length of the z-chunks a stage launch is cut into, chosen by grid size
and CTAs per SM, changes nothing but the launch shape: states are bitwise
those of fixed chunks, reductions the same sums in another order."""
from __future__ import annotations

import os

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def run(rp, psi0, zc):
    old = os.environ.get("GPE_ZC")
    if zc:
        os.environ["GPE_ZC"] = str(zc)
    try:
        s = Solver(rp)
    finally:
        if old is None:
            os.environ.pop("GPE_ZC", None)
        else:
            os.environ["GPE_ZC"] = old
    s.set_state(psi0)
    info = s.solver(5, want_norm=True, want_energy=True)
    out, e = s.get_state(), s.energy()
    s.close()
    return out, info, e


# one plane per CTA, chunks that divide nz, a last chunk of one plane, several rounds
@pytest.mark.parametrize("shape", [(6, 6, 6), (33, 9, 25), (64, 64, 64), (70, 81, 47), (160, 96, 61)])
@pytest.mark.parametrize("storage", ["c128", "c64"])
@pytest.mark.parametrize("scheme,order", [("rk4", 4), ("rk4", 2), ("rk45", 4), ("euler", 2)])
def test_states_do_not_depend_on_the_chunks(gpu, shape, storage, scheme, order):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.002,
                   scheme=scheme, eqn_to_solve=4, bcs=2, order=order, g=1.0, mu=2.0, omx=0.1, storage=storage)
    rng = np.random.default_rng(nx + ny + nz)
    psi0 = 1.0 + 0.2 * (rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx)))
    ref, iref, eref = run(rp, psi0, 5)
    out, info, e = run(rp, psi0, 0)
    np.testing.assert_array_equal(out, ref)
    # sums of nx ny nz terms in two orders: at most n eps apart
    tol = nx * ny * nz * 2.3e-16
    assert info.norm == pytest.approx(iref.norm, rel=tol)
    assert info.energy == pytest.approx(iref.energy, rel=tol) and e == pytest.approx(eref, rel=tol)
    assert (info.t, info.dt_re, info.errmax) == (iref.t, iref.dt_re, iref.errmax)


@pytest.mark.parametrize("eqn", [1, 2, 3])
@pytest.mark.parametrize("bcs,order", [(1, 4), (1, 2), (2, 4)])
@pytest.mark.parametrize("storage", ["c128", "c64"])
def test_small_grid_kernel_equals_the_march(gpu, eqn, bcs, order, storage):
    # 35 x 22 x 13 is a small grid (one thread per site); any chunk asked for selects the march
    rp = RunParams(nx=35, ny=22, nz=13, xr=4.25, yr=2.625, zr=1.5, tau=0.001, scheme="rk4", eqn_to_solve=eqn, bcs=bcs,
                   order=order, Urhs=0.2, diss_amp=0.1 if eqn != 2 else 0.0, storage=storage)
    rng = np.random.default_rng(eqn + 10 * bcs + order)
    psi0 = 1.0 + 0.3 * (rng.normal(size=(13, 22, 35)) + 1j * rng.normal(size=(13, 22, 35)))
    ref, _, _ = run(rp, psi0, 4)
    out, _, _ = run(rp, psi0, 0)
    np.testing.assert_array_equal(out, ref)
