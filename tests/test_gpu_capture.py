"""Steps enqueued on a handle's stream while its owner captures that stream:
one or two at a time are plain launches, with a norm too, whatever the handle
has done before."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpe_b200.solver import RunParams, Solver

pytestmark = pytest.mark.gpu


# 20 x 18 x 16 one thread per site; 72 x 70 x 66 the march
@pytest.mark.parametrize("shape", [(20, 18, 16), (72, 70, 66)])
@pytest.mark.parametrize("scheme", ["rk4", "rk2"])
@pytest.mark.parametrize("norm", [False, True])
def test_steps_under_the_callers_capture(gpu, shape, scheme, norm):
    nx, ny, nz = shape
    rp = RunParams(nx=nx, ny=ny, nz=nz, xr=0.25 * (nx - 1), yr=0.25 * (ny - 1), zr=0.25 * (nz - 1), tau=0.004,
                   scheme=scheme, eqn_to_solve=2, bcs=1, order=4)
    rng = np.random.default_rng(3)
    psi0 = 1.0 + 0.1 * (rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx)))
    with Solver(rp) as one:
        one.set_state(psi0)
        for _ in range(7):
            one.solver(1)
        want = one.get_state()
    with Solver(rp) as s:
        s.set_state(psi0)
        s.solver(1, want_norm=norm, wait=False)  # the kernels are loaded, the dt is known
        s.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.ExternalStream(s.stream())):
            graph.capture_begin(capture_error_mode="thread_local")
            try:
                s.solver(1, want_norm=norm, wait=False)
                s.solver(2, want_norm=norm, wait=False)
            finally:
                graph.capture_end()
            graph.replay()
            graph.replay()
        s.sync()
        np.testing.assert_array_equal(s.get_state(), want)
        assert s.solver(1, want_norm=True).norm > 0.0
        del graph
