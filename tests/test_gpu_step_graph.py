"""A call of many fixed steps replays captured graphs of eight steps and of
one, whose stage kernels are launched as dependents of each other; states and
clock equal those of one call per step, bitwise, for every remainder."""
from __future__ import annotations

import numpy as np
import pytest

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


# (20, 18, 16) one thread per site; (72, 70, 66) the march, several CTAs per SM
@pytest.mark.parametrize("shape", [(20, 18, 16), (72, 70, 66)])
@pytest.mark.parametrize("storage,scheme", [("c128", "rk4"), ("c64", "rk4"), ("c128", "rk2")])
def test_many_steps_equal_single_calls(gpu, shape, storage, scheme):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.004,
                   scheme=scheme, eqn_to_solve=2, bcs=1, order=4, Urhs=0.1, storage=storage)
    rng = np.random.default_rng(nx)
    psi0 = 1.0 + 0.1 * (rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx)))
    one, many = Solver(rp), Solver(rp)
    one.set_state(psi0)
    many.set_state(psi0)
    for n in (2, 3, 8, 9, 10, 11, 17, 18, 25):
        for _ in range(n - 1):
            one.solver(1)
        a = one.solver(1, want_norm=n % 2 == 0)
        b = many.solver(n, want_norm=n % 2 == 0)
        np.testing.assert_array_equal(many.get_state(), one.get_state(), err_msg=f"{n} steps")
        assert (one.t, one.p) == (many.t, many.p) and b.accepted == n
        if n % 2 == 0:
            assert a.norm == b.norm
    one.close()
    many.close()


def test_changing_time_steps(gpu):
    # graphs belong to a dt: each comes back, changes after one call, and
    # alternates from call to call, with and without a norm
    rp = RunParams(nx=20, ny=18, nz=16, xr=4.75, yr=4.25, zr=3.75, tau=0.004, scheme="rk4", eqn_to_solve=2, bcs=1, order=4)
    rng = np.random.default_rng(7)
    psi0 = 1.0 + 0.1 * (rng.normal(size=(16, 18, 20)) + 1j * rng.normal(size=(16, 18, 20)))
    one, many = Solver(rp), Solver(rp)
    one.set_state(psi0)
    many.set_state(psi0)
    for n, dt, norm in [(10, 4e-3, True), (10, 4e-3, True), (10, 2e-3, True), (1, 4e-3, True), (1, 4e-3, True),
                        (1, 2e-3, True), (1, 4e-3, True), (40, 2e-3, False), (9, 4e-3, False), (9, 2e-3, True)]:
        one.dt = many.dt = complex(dt, 0.0)
        for _ in range(n):
            one.solver(1)
        b = many.solver(n, want_norm=norm)
        np.testing.assert_array_equal(many.get_state(), one.get_state(), err_msg=f"{n} steps of {dt}")
        assert one.t == many.t
        if norm:
            assert b.norm == pytest.approx(one.get_norm(), rel=16 * 18 * 20 * 2.3e-16)
    one.close()
    many.close()


# (the shapes march, and their norm and energy launches have more blocks than
# the last stage; complex64 has the layout of two sites a thread)
@pytest.mark.parametrize("n,storage", [(96, "c128"), (128, "c64")])
@pytest.mark.parametrize("scheme", ["rk4", "rk2"])
def test_other_reductions_between_steps_with_a_norm(gpu, n, storage, scheme):
    # a captured step with a norm keeps the address of its block partials:
    # other reductions of the handle, and a second handle's memory, leave it
    # as it is
    h = 0.25 * (n - 1)
    rp = RunParams(nx=n, ny=n, nz=n, xr=h, yr=h, zr=h, tau=0.004, scheme=scheme, eqn_to_solve=2, bcs=1, order=4,
                   storage=storage)
    rng = np.random.default_rng(n)
    psi0 = 1.0 + 0.1 * (rng.normal(size=(n, n, n)) + 1j * rng.normal(size=(n, n, n)))
    with Solver(rp) as s:  # alone: plain steps, no reduction before the last
        s.set_state(psi0)
        for _ in range(5):
            s.solver(1)
        alone, norm_alone = s.get_state(), s.get_norm()
        s.set_state(psi0)
        s.solver(1)
        second_alone = s.get_state()
    first = Solver(rp)
    first.set_state(psi0)
    first.solver(1, want_norm=True)
    first.solver(1, want_norm=True)
    first.get_norm()
    first.energy()
    second = Solver(rp)
    second.set_state(psi0)
    first.solver(1, want_norm=True)
    first.solver(1, want_energy=True)
    norm = first.solver(1, want_norm=True).norm
    second.solver(1)
    np.testing.assert_array_equal(second.get_state(), second_alone)
    np.testing.assert_array_equal(first.get_state(), alone)
    # sums of n^3 non-negative terms in two orders: at most n^3 eps apart
    assert norm == pytest.approx(first.get_norm(), rel=n ** 3 * 2.3e-16)
    assert first.get_norm() == norm_alone
    first.close()
    second.close()
