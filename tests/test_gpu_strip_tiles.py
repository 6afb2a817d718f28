"""The strip product's tiles (k_strip.cu): 8-row strips on FP64 matrix
instructions (32 and 112 columns per warp) and the flat mapping over strips
(FP32, and strips of 2 and 4 rows), at the edges of their widths, with a
ragged last strip, empty rows and a last row alone in its strip."""
import numpy as np
import pytest
import scipy.sparse as sp

import lgh_b200 as L

pytestmark = pytest.mark.gpu

EPS64, EPS32 = 2.0 ** -53, 2.0 ** -24


def _banded(n, seed):
    """Rows of 0 to 11 entries within 9 of the diagonal: an 8-row strip's
    union holds at most 26 columns."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(0, 12, size=n)
    cnt[n - 1] = 3
    rows = np.repeat(np.arange(n), cnt)
    cols = np.clip(rows + rng.integers(-9, 10, size=rows.size), 0, n - 1)
    A = sp.csr_matrix((rng.standard_normal(rows.size), (rows, cols)), (n, n))
    A.sum_duplicates()
    return A


def _check(A, X, fp32, R):
    csr = dict(n=A.shape[0], rowptr=A.indptr.astype(np.int64),
               colidx=A.indices.astype(np.int32), vals=A.data)
    Y, used = L.test_spmm_strip(L.Mat(csr), X, fp32=fp32, R=R)
    assert used == R
    # at most 26 products summed in any order, and in FP32 the rounding of
    # the value, of X and of nothing else: (26 + 2) u |A| |X| per element
    u = EPS32 if fp32 else EPS64
    bound = 28 * u * (abs(A) @ np.abs(X)) * (1 + 1e-3)
    assert np.all(np.abs(Y - A @ X) <= bound + (26 + 2) * EPS64
                  * (abs(A) @ np.abs(X)))


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("R", [2, 4, 8])
@pytest.mark.parametrize("w", [1, 2, 5, 31, 32, 33, 63, 129])
def test_strip_widths(w, R, fp32):
    A = _banded(1001, 7 * w + R)
    X = np.random.default_rng(w).standard_normal((1001, w))
    _check(A, X, fp32, R)


@pytest.mark.parametrize("n,w", [(19001, 100), (19001, 112), (19001, 113),
                                 (9601, 219), (9601, 224), (18000, 112)])
def test_strip_wide_tile(n, w):
    A = _banded(n, n + w)
    X = np.random.default_rng(w).standard_normal((n, w))
    _check(A, X, False, 8)


@pytest.mark.parametrize("R,w", [(2, 1030), (4, 513), (8, 1030)])
def test_strip_wider_than_one_launch(R, w):
    """More packs than one launch's threads cover."""
    A = _banded(203, R)
    X = np.random.default_rng(w).standard_normal((203, w))
    _check(A, X, False, R)
    if R == 8:
        _check(A, X, True, R)
