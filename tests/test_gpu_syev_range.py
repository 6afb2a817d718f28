"""The eigensolver over the exponent range: matrices scaled by powers of two
up to the last binade (the scaled problem has the same rotations, so the
eigenvalues agree with the unscaled ones to rounding, as in
test_gpu_syev_blocks.py 1e-13 of the norm), and the sweeps it takes on
spectra that lose many digits: a sweep count at the limit of 40 would be an
unconverged result."""

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 20, 50])
@pytest.mark.parametrize("e", [0, -900, 900, 1023])
def test_scaled(cuda_device, n, e):
    """Largest diagonal entry 1.5 2^e: at 1023 differences and diagonal are
    in the last binade, sums of a row below the overflow limit."""
    rng = np.random.default_rng(n)
    A = 1e-3 / n * rng.standard_normal((n, n))
    A = 0.5 * (A + A.T)
    A[np.arange(n), np.arange(n)] = np.linspace(0.01, 1.5, n)
    ref = np.linalg.eigvalsh(A)
    w, V, sweeps = L.test_syev(np.ldexp(A, e))
    assert np.max(np.abs(np.sort(np.ldexp(w, -e)) - ref)) <= 1e-13 * np.linalg.norm(A)
    assert np.max(np.abs(V.T @ V - np.eye(n))) < 1e-12
    assert sweeps < 20


@pytest.mark.parametrize("n", [33, 220])
def test_converges(cuda_device, n):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    i = np.arange(n)
    spectra = {
        "low rank": np.where(i < n // 3, 1.0 / (1 + i), 0.0),
        "plus and minus": np.where(i % 2 == 0, 1.0, -1.0),
        "decay to 1e-9": np.logspace(0, -9, n),
    }
    for name, lam in spectra.items():
        A = (Q * lam) @ Q.T
        w, _, sweeps = L.test_syev(0.5 * (A + A.T))
        assert np.max(np.abs(np.sort(w) - np.sort(lam))) < 1e-13 * np.linalg.norm(lam), name
        assert sweeps < 40, name
    d = np.logspace(0, -6, n)
    H = np.eye(n) + 0.02 / np.sqrt(n) * rng.standard_normal((n, n))
    w, _, sweeps = L.test_syev(0.5 * (H + H.T) * d[:, None] * d[None, :])
    assert sweeps < 15
