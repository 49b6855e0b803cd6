"""gpe_norm_noalloc cuts each plane into parts and walks rows in pairs; sizes
at the edges of both, against the quadrature in numpy."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def weights(n):
    w = np.ones(n)
    w[[0, n - 1]], w[[1, n - 2]], w[[2, n - 3]] = 3 / 8, 7 / 6, 23 / 24
    return w


# rows below, at and past a part; one row pair and an odd row; many planes (one part); long rows
@pytest.mark.parametrize("shape", [(6, 6, 6), (33, 8, 7), (31, 9, 11), (64, 17, 6), (100, 300, 6), (7, 64, 2100),
                                   (9, 10, 8192), (1030, 7, 9)])
@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_split_planes(gpu, shape, dtype):
    import torch

    from gpe_b200 import _lib as L

    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny + nz)
    psi = (rng.normal(size=(nz, ny, nx)) + 1j * rng.normal(size=(nz, ny, nx))).astype(
        np.complex64 if dtype == "c64" else np.complex128)
    d_psi, out = torch.from_numpy(psi).cuda(), torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
    rc = L.load().gpe_norm_noalloc(C.c_void_p(d_psi.data_ptr()), L.GPE_C64 if dtype == "c64" else L.GPE_C128, nx, ny,
                                   nz, 0.5, 0.25, 2.0, C.c_void_p(out.data_ptr()),
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == L.GPE_OK
    v = np.abs(psi.astype(np.complex128)) ** 2
    ref = np.einsum("kji,k,j,i->", v, weights(nz), weights(ny), weights(nx)) * 0.25
    # terms of one sign: at most n eps apart
    assert out.item() == pytest.approx(ref, rel=nx * ny * nz * 2.3e-16)
