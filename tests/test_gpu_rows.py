"""Layout kernels that take a warp per row (packing, unpacking, ghost cells,
the random-phase state): row lengths around the 32-lane and four-chunk
boundaries, both storages and element types of the host array."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200 import ic
from gpe_b200.pool import Pool
from gpe_b200.solver import RunParams, Solver
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [6, 31, 32, 33, 127, 129, 260])
@pytest.mark.parametrize("storage", ["c128", "c64"])
@pytest.mark.parametrize("bcs,order", [(1, 4), (2, 4), (1, 2), (2, 2)])
def test_pack_ghosts_unpack(gpu, nx, storage, bcs, order):
    ny, nz = 7, 6
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=1.5, zr=1.25, tau=0.002, scheme="rk4", eqn_to_solve=4,
                   bcs=bcs, order=order, storage=storage)
    rng = np.random.default_rng(nx + bcs)
    psi = rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx))
    ct = np.complex64 if storage == "c64" else np.complex128
    s = Solver(rp)
    for t in (np.complex128, np.complex64):
        s.set_state(psi.astype(t))
        np.testing.assert_array_equal(s.get_state(), psi.astype(t).astype(ct).astype(np.complex128))
        np.testing.assert_array_equal(s.get_state(np.complex64), psi.astype(t).astype(np.complex64))
    # every ghost enters the energy's Laplacian (sum of n terms of both signs, each a few eps of its scale)
    held = s.get_state()
    e = s.energy()
    ref = Oracle(rp.replace(storage="c128", compute="auto")).energy(held)
    scale = np.sum(np.abs(held) ** 2) * 400.0 * 0.125
    assert abs(e - ref) <= scale * (1e-13 if storage == "c128" else 1e-6)
    # the pool packs its copy of the interior: one step equals the handle's, bitwise
    pool = Pool(Pool.solve_bytes(rp) + (32 << 20))
    assert pool.submit(rp, held.astype(ct), 1, 0)
    (r,) = pool.run_all()
    pool.close()
    s.solver(1)
    np.testing.assert_array_equal(r.psi, s.get_state(ct))
    s.close()


@pytest.mark.parametrize("shape", [(33, 6, 7), (6, 40, 9), (130, 12, 6)])
def test_random_phase_rows(gpu, shape):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), bcs=1, order=4)
    s = Solver(rp)
    s.set_ic(ic.device_spec("random_phase", seed=5, kc=2.5))
    ref = ic.random_phase(rp, seed=5, kc=2.5)
    assert np.linalg.norm(s.get_state() - ref) <= 1e-12 * np.linalg.norm(ref)
    s.close()
