"""The block Jacobi eigensolver at the edges of its blocks (one entry, one
block, one pair, a partial last block, odd sizes), on spectra that rotate
little or not at all (diagonal, zero, repeated eigenvalues, plus/minus
pairs), and on a graded one.  Bounds: backward stability with a few dozen
sweeps' roundings, 1e-13 of the norm for eigenvalues as the scalar ordering
is held to, 1e-12 for orthogonality."""

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu


def _check(A):
    n = A.shape[0]
    w, V, sweeps = L.test_syev(A)
    nrm = max(np.linalg.norm(A), 1e-300)
    ref = np.linalg.eigvalsh(A)
    assert np.max(np.abs(np.sort(w) - ref)) <= 1e-13 * nrm
    assert np.max(np.abs(V.T @ V - np.eye(n))) < 1e-12
    assert np.max(np.abs(A @ V - V * w)) <= 1e-12 * nrm
    assert 0 <= sweeps <= 40
    return w, sweeps


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 47, 64, 65, 97,
                               131, 220, 301, 520])
def test_random(cuda_device, n):
    A = np.random.default_rng(n).standard_normal((n, n))
    w, sweeps = _check(A + A.T)
    assert sweeps <= 14


@pytest.mark.parametrize("n", [5, 32, 50, 129])
def test_special(cuda_device, n):
    rng = np.random.default_rng(n)
    _check(np.zeros((n, n)))
    d = rng.standard_normal(n)
    w, _ = _check(np.diag(d))
    assert np.array_equal(np.sort(w), np.sort(d))
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    for lam in (np.where(np.arange(n) % 2 == 0, 1.0, -1.0),
                np.repeat([3.0, 3.0, -3.0, 1e-9, 0.0], n)[:n],
                np.linspace(1.0, 1.001, n)):
        A = (Q * lam) @ Q.T
        _check(0.5 * (A + A.T))


@pytest.mark.parametrize("n", [60, 200])
def test_graded(cuda_device, n):
    """A scaled diagonally dominant matrix keeps its small eigenvalues to
    high relative accuracy under the relative rotation threshold."""
    rng = np.random.default_rng(n)
    H = np.eye(n) + 0.02 / np.sqrt(n) * rng.standard_normal((n, n))
    H = 0.5 * (H + H.T)
    d = np.logspace(0, -6, n)
    A = H * d[:, None] * d[None, :]
    w, _, _ = L.test_syev(A)
    # the eigenvalues of D H D, to relative accuracy, from its inverse's
    # largest ones
    inv = np.linalg.inv(H) / d[:, None] / d[None, :]
    small = 1.0 / np.sort(np.linalg.eigvalsh(0.5 * (inv + inv.T)))[::-1][:5]
    assert np.max(np.abs(np.sort(w)[:5] - small) / small) < 1e-10
