"""The shifts of a batched operation in device, pinned and pageable
memory, written by work that is still queued on the default stream when the
call is made: the call takes the written values."""

import ctypes

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu

SHIFTS = [0.25, 1.5, 7.0]


@pytest.fixture(scope="module")
def glr(cuda_device):
    side = 37
    mass = P.lumped_mass(side, 2)
    mat = L.Mat(P.z_operator(side, 2, 25.0, mass))
    prior = L.Prior(Z=mat, mass=mass)
    n = side * side
    A = np.random.default_rng(4).standard_normal((n, 20))
    B = L.Mat(dense=A @ A.T / n)
    g = L.Glr(B, prior, L.glr_opts(ell=20, seed=0, check=0))
    X = np.random.default_rng(5).standard_normal((n, 2))
    return n, g, X, np.concatenate(g.solve_batch(SHIFTS, X), axis=1)


@pytest.mark.parametrize("where", ["device", "pinned", "pageable"])
def test_queued_shifts(glr, where):
    import torch
    n, g, X, ref = glr
    m, ns = X.shape[1], len(SHIFTS)
    src = torch.tensor(SHIFTS, dtype=torch.float64, device="cuda")
    c = torch.full((ns,), 3.0, dtype=torch.float64,
                   device="cuda" if where == "device" else "cpu",
                   pin_memory=where == "pinned")
    bx, by = L.DeviceBlock(n, m, X), L.DeviceBlock(n, m * ns)
    big = torch.ones(8192, 8192, device="cuda")
    out = torch.empty_like(big)
    torch.mm(big, big, out=out)             # loads the library
    torch.cuda.synchronize()
    for _ in range(10):                     # some 0.1 s of queued work
        torch.mm(big, big, out=out)
    c.copy_(src, non_blocking=True)
    rc = L.load().lgh_glr_solve_batch(
        g.h, ns, ctypes.cast(c.data_ptr(), L.c_dbl_p), m, bx.ptr(), n,
        by.ptr(), n)
    assert rc == 0
    assert np.array_equal(by.get(), ref)
