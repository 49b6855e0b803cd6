"""Norms of pooled solves that join and leave between calls of one step each:
every result's norm is that of its own final state, RK4 and RKF45 (whose state
changes its field with every accepted step), both storages."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.pool import Pool
from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


def params(n, scheme, storage):
    h = 0.25 * (n - 1)
    return RunParams(nx=n, ny=n + 1, nz=n + 2, xr=h, yr=h, zr=h, tau=0.002, scheme=scheme, eqn_to_solve=4, bcs=2,
                     order=4, mu=2.0, omx=0.1, storage=storage)


def test_each_norm_is_its_own_states(gpu):
    rng = np.random.default_rng(5)
    solves = []
    for k, (n, scheme, storage, steps) in enumerate([
            (17, "rk4", "c64", 1), (24, "rk45", "c64", 3), (9, "rk45", "c128", 2), (31, "rk4", "c64", 4),
            (12, "rk4", "c128", 3), (20, "rk45", "c64", 1), (15, "rk45", "c128", 4), (33, "rk4", "c128", 2)]):
        p = params(n, scheme, storage)
        psi = 1.0 + 0.1 * (rng.normal(size=(n + 2, n + 1, n)) + 1j * rng.normal(size=(n + 2, n + 1, n)))
        solves.append((k, p, psi, steps))
    pool = Pool(sum(Pool.solve_bytes(p) for _, p, _, _ in solves) + (1 << 20))
    waiting, got = list(solves), []
    while waiting or len(got) < len(solves):
        for k, p, psi, steps in waiting[:2]:  # two more join before every step
            assert pool.submit(p, psi, steps, k)
        del waiting[:2]
        pool.step(1)
        got += pool.poll()
    assert sorted(r.tag for r in got) == [k for k, _, _, _ in solves]
    for r in got:
        k, p, _, steps = solves[r.tag]
        assert r.steps == steps and r.status == 0
        with Solver(p) as s:
            s.set_state(r.psi)
            # sums of terms of one sign (but for the weights) in two orders
            assert r.norm == pytest.approx(s.get_norm(), rel=r.psi.size * 2.3e-16)
    pool.close()
