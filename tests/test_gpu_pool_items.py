"""A pool cuts its solves into work items by how much work the class holds,
and forms norms in a pass of their own: states and norms are the same whatever
else is in the pool, and states those of the single-solve handle."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.pool import Pool
from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def params(n, scheme, storage, order):
    nx, ny, nz = n
    kw = dict(mu=10.0, omx=0.05, gamma=0.05) if scheme == "rk45" else dict(mu=1.0)
    return RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.004,
                     scheme=scheme, eqn_to_solve=4, bcs=2, order=order, g=1.0, storage=storage, **kw)


def state(rp, seed):
    rng = np.random.default_rng(seed)
    shape = (rp.nz, rp.ny, rp.nx)
    psi = 3.0 * (rp.scheme == "rk45") + 1.0 + 0.1 * (rng.normal(size=shape) + 1j * rng.normal(size=shape))
    return psi.astype(np.complex64 if rp.storage == "c64" else np.complex128)


def run(solves, steps, max_steps):
    pool = Pool(sum(Pool.solve_bytes(rp) for rp, _ in solves) + (64 << 20))
    for k, (rp, psi) in enumerate(solves):
        assert pool.submit(rp, psi, steps, k)
    res = {r.tag: r for r in pool.run_all(max_steps=max_steps)}
    pool.close()
    return [res[k] for k in range(len(solves))]


# 1 solve (short items), 17 and 20 (parameters of more than 16 solves), a chosen item length
@pytest.mark.parametrize("count", [1, 17, 20])
@pytest.mark.parametrize("scheme,storage,order", [("rk4", "c64", 4), ("rk4", "c128", 2), ("rk45", "c128", 4),
                                                  ("rk45", "c64", 2)])
def test_items_follow_the_class(gpu, count, scheme, storage, order):
    shapes = [(40, 33, 35), (9, 8, 66), (64, 30, 7), (33, 17, 21)]
    rps = [params(shapes[k % 4], scheme, storage, order) for k in range(count)]
    if count > 1:
        rps[1] = rps[1].replace(tile_zc=5)
    solves = [(rp, state(rp, k)) for k, rp in enumerate(rps)]
    res = run(solves, 6, 4)
    for k in sorted({0, 1 % count, 2 % count, count - 1}):
        rp, psi = solves[k]
        (alone,) = run([(rp.replace(tile_zc=0), psi)], 6, 6)
        np.testing.assert_array_equal(res[k].psi, alone.psi)
        assert res[k].norm == alone.norm and res[k].t == alone.t and res[k].dt == alone.dt
        s = Solver(rp)
        s.set_state(psi)
        s.solver(6)
        np.testing.assert_array_equal(res[k].psi, s.get_state(psi.dtype))
        # the same terms of one sign in another order: n eps
        assert res[k].norm == pytest.approx(s.get_norm(), rel=rp.nx * rp.ny * rp.nz * 2.3e-16)
        s.close()
