"""The spectral sums fold each axis onto its distinct squared distances; odd,
even and short axes fold differently.  Against the numpy oracle."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver
from oracle import fft_diag as D

pytestmark = pytest.mark.gpu


# shortest axes, one lane past a 32-lane chunk, odd and even extents, a long x axis
@pytest.mark.parametrize("shape", [(6, 6, 6), (7, 6, 9), (8, 13, 11), (62, 7, 6), (63, 6, 8), (65, 20, 66), (259, 9, 8)])
@pytest.mark.parametrize("storage", ["c128", "c64"])
def test_folded_spectra_match_oracle(gpu, shape, storage):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), bcs=1, order=4,
                   storage=storage)
    rng = np.random.default_rng(nx + 7 * ny + nz)
    s = Solver(rp)
    s.set_state(1 + rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx)))
    psi = s.get_state()
    dev = s.condensed(spectrum=True)
    plain = s.condensed()
    out = s.filtered(3.0, m=0.7)
    s.close()
    rec, a = D.condensed_particles(psi, rp.xr, rp.yr, rp.zr)
    eta, nharm, F = D.spectrum(a)
    # sums of at most n terms of one sign, each good to a few eps (the transform: log2 n of them)
    tol = (nx * ny * nz + 50) * 2.3e-16
    for k, v in rec.items():
        assert dev[k] == pytest.approx(v, rel=tol), k
        assert plain[k] == dev[k], k
    assert np.array_equal(dev["nharm"], nharm)
    np.testing.assert_allclose(dev["eta"], eta, rtol=tol)
    np.testing.assert_allclose(dev["F"], F, rtol=tol)
    ref = D.filtered_surface(a, 0.7, 3.0)
    assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)
