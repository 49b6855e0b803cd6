"""What a handle's launch options (tile_zc, GPE_TILE, GPE_ZC) may change: the
shape of its launches, nothing in the states."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def params(shape, **kw):
    nx, ny, nz = shape
    d = dict(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.002, scheme="rk4",
             eqn_to_solve=2, bcs=1, order=4)
    d.update(kw)
    return RunParams(**d)


def noise(shape, seed):
    rng = np.random.default_rng(seed)
    s = shape[::-1]
    return 1.0 + 0.2 * (rng.normal(size=s) + 1j * rng.normal(size=s))


# a chunk asked for together with the layout that has one thread per site and no chunks
@pytest.mark.parametrize("zc", [1, 4, 100])
@pytest.mark.parametrize("scheme", ["rk4", "rk45"])
def test_a_thread_per_site_updates_every_plane(gpu, monkeypatch, zc, scheme):
    shape = (35, 22, 13)
    psi0 = noise(shape, 1)
    out = []
    for tile, chunk in [(None, 5), ("1", zc)]:
        with monkeypatch.context() as m:
            if tile:
                m.setenv("GPE_TILE", tile)
            s = Solver(params(shape, scheme=scheme, tile_zc=chunk))
        s.set_state(psi0)
        info = s.solver(5)
        out.append((s.get_state(), info.errmax, s.dt))
        s.close()
    np.testing.assert_array_equal(out[1][0], out[0][0])
    assert out[1][1:] == out[0][1:]


# the partition of a launch fixes the order of its sums, so equal norms of
# eight states say that both handles cut their launches alike
@pytest.mark.parametrize("storage", ["c128", "c64"])
def test_the_environment_counts_when_a_handle_is_created(gpu, monkeypatch, storage):
    shape = (96, 96, 96)
    norms = []
    for keep in (True, False):
        monkeypatch.setenv("GPE_ZC", "17")
        s = Solver(params(shape, storage=storage))
        if not keep:
            monkeypatch.delenv("GPE_ZC")
        row = []
        for seed in range(8):
            s.set_state(noise(shape, seed))
            row.append(s.solver(1, want_norm=True).norm)
        norms.append(row)
        s.close()
    assert norms[0] == norms[1]
