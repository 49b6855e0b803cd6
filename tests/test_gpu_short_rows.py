"""Grids whose rows are shorter than a warp, or few: the layout kernels, the
diagnostics, the norm and the initial states take their sites one by one, and
give what they give elsewhere."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200 import ic
from gpe_b200.solver import RunParams, Solver
from oracle import fft_diag as D

pytestmark = pytest.mark.gpu

# 6 to 48 sites a row, on both sides of 8, 16, 32 and 48; few long rows; few columns
SHAPES = [(6, 70, 9), (8, 9, 70), (9, 33, 17), (16, 40, 40), (17, 40, 40), (31, 41, 40), (32, 41, 40), (33, 41, 40),
          (47, 80, 70), (48, 80, 70), (700, 6, 8), (6, 6, 333), (13, 15, 50)]


def params(shape, **kw):
    nx, ny, nz = shape
    d = dict(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.002, scheme="rk4",
             eqn_to_solve=2, bcs=1, order=4, mu=2.0, omx=0.1, omy=0.2, omz=0.05)
    d.update(kw)
    return RunParams(**d)


def noise(shape, seed):
    rng = np.random.default_rng(seed)
    s = shape[::-1]
    return 1.0 + 0.2 * (rng.normal(size=s) + 1j * rng.normal(size=s))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage,dtype", [("c128", np.complex128), ("c64", np.complex64), ("c128", np.complex64)])
@pytest.mark.parametrize("bcs", [1, 2])
def test_states_go_in_and_out(gpu, shape, storage, dtype, bcs):
    psi = noise(shape, 1).astype(dtype)
    with Solver(params(shape, storage=storage, bcs=bcs)) as s, Solver(params(shape, storage=storage, bcs=bcs)) as t:
        s.set_state(psi)
        np.testing.assert_array_equal(s.get_state(dtype=dtype), psi)
        # ghosts written by the layout kernel against those a stage wrote
        t.set_state(psi)
        t.solver(1)
        s.set_state(t.get_state())
        s.solver(1)
        t.solver(1)
        np.testing.assert_array_equal(s.get_state(), t.get_state())


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["c128", "c64"])
def test_diagnostics(gpu, shape, storage):
    rp = params(shape, storage=storage)
    tol = 1e-12  # that of the diagnostics' own tests
    with Solver(rp) as s:
        s.set_state(noise(shape, 2))
        psi = s.get_state().astype(np.complex128)
        rec, a = D.condensed_particles(psi, rp.xr, rp.yr, rp.zr)
        eta, nharm, F = D.spectrum(a)
        scale = np.sum(np.abs(psi) ** 2)
        for spectrum in (True, False):
            dev = s.condensed(spectrum=spectrum)
            for k in ("M", "tot", "temp", "temp2", "H", "mass_density"):
                assert dev[k] == pytest.approx(rec[k], rel=tol), k
            assert abs(dev["n0"] - rec["n0"]) <= tol * scale
        dev = s.condensed(spectrum=True)
        assert np.array_equal(dev["nharm"], nharm)
        np.testing.assert_allclose(dev["eta"], eta, rtol=tol, atol=tol * scale / psi.size)
        np.testing.assert_allclose(dev["F"], F, rtol=tol, atol=tol * scale)
        ref = D.filtered_surface(a, 1.0, 4.0)
        assert np.linalg.norm(s.filtered(4.0) - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["c128", "c64"])
def test_initial_states(gpu, shape, storage):
    rp = params(shape, storage=storage, bcs=2)
    eps = 1e-13 if storage == "c128" else 1e-13 + 2.0 ** -24  # the closed forms' own, and a rounding to storage
    line = dict(x0=0.1, y0=0.2, z0=0.15)
    for names, kw, ref in [
            (("fermi", "line_pade"), dict(line=dict(line, dir="z")),
             lambda: ic.fermi(rp) * ic.vortex_line_pade(rp, **line, dir="z")),
            (("line",), dict(line=dict(line, dir="x")), lambda: ic.vortex_line(rp, **line, dir="x")),
            (("random_phase",), dict(seed=3, kc=1.5), lambda: ic.random_phase(rp, seed=3, kc=1.5))]:
        with Solver(rp) as s:
            s.set_ic(ic.device_spec(*names, **kw))
            want = ref()
            bar = (1e-12 + eps if names == ("random_phase",) else eps) * max(1.0, float(np.abs(want).max()))
            np.testing.assert_allclose(s.get_state(), want, rtol=0, atol=bar)
            e = s.energy()
            with Solver(rp) as t:  # the ghosts are those of a packed state
                t.set_state(s.get_state())
                assert t.energy() == e
