"""The eigensolver's rounding on the spectra that a randomized build meets,
decaying and rank-deficient ones.

Orthogonality: a column of V takes part in n rotations a sweep, each off by
an eps = 1.1e-16 in its scale; over 30 sweeps their random sum is eps sqrt
(30 n) a column, eps n sqrt (30) over the matrix, and three times that is
the bound (n = 220: 4e-13).  Eigenvalues: Rayleigh quotients in FP64 against
those of LAPACK's vectors in long double, whose own error is the square of
the vectors': ten eps of the norm."""

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _spectra(n):
    i = np.arange(n)
    return {
        "decay": np.logspace(0, -12, n),
        "low rank": np.where(i < n // 3, 1.0 / (1 + i), 0.0),
        "plus and minus": np.where(i % 2 == 0, 1.0, -1.0),
    }


@pytest.mark.parametrize("n", [20, 33, 64, 131, 220])
@pytest.mark.parametrize("name", sorted(_spectra(4)))
def test_rounding(cuda_device, name, n):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * _spectra(n)[name]) @ Q.T
    A = 0.5 * (A + A.T)
    w, V, _ = L.test_syev(A)
    U = np.linalg.eigh(A)[1].astype(np.longdouble)
    ref = (U * (A.astype(np.longdouble) @ U)).sum(0) / (U * U).sum(0)
    nrm = np.linalg.norm(A)
    assert np.linalg.norm(V.T @ V - np.eye(n)) < 3 * EPS * n * np.sqrt(30)
    assert np.linalg.norm(np.sort(w) - np.sort(ref.astype(float))) < 10 * EPS * nrm
