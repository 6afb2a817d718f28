"""Cholesky and triangular inverse at the edges of their panels (16 columns)
and register columns (32 T rows, above 512 through shared memory), and a
failure in a later panel.

The matrix is X X^T + n I with condition below 10, so the factor and its
inverse are good to n u cond, 1e-12 at the largest size."""

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu


def _spd(n):
    X = np.random.default_rng(n).standard_normal((n, n)) / np.sqrt(n)
    return X @ X.T + np.eye(n)


@pytest.mark.parametrize("n", [1, 7, 15, 16, 17, 32, 33, 64, 65, 127, 129, 256,
                               257, 511, 512, 513])
def test_panels(cuda_device, n):
    G = _spd(n)
    Lc, Li, info = L.test_potrf(G)
    assert info[0] == 0 and info[1] == 0
    ref = np.linalg.cholesky(G)
    assert np.max(np.abs(np.tril(Lc) - ref)) < 1e-12
    assert np.max(np.abs(np.tril(Li) @ ref - np.eye(n))) < 1e-12
    assert not np.triu(Li, 1).any()


@pytest.mark.parametrize("bad", [3, 20, 36])
def test_failure_position(cuda_device, bad):
    """A negative pivot in the first, second and last (short) panel."""
    G = _spd(37)
    G[bad, bad] = -1.0
    _, Li, info = L.test_potrf(G)
    assert info[0] != 0 and Li is None
