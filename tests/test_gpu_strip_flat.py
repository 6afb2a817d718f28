"""Strips of 2 and 4 rows with four packs per thread, which only many strips
take: at the edges of the packs (32 | 33 with 2 rows, 24 | 26 with 4, ragged
last packs), with a ragged last strip and empty rows, and on operators whose
rows share no column (the strip height 2 is the cost model's own choice
there)."""

import numpy as np
import pytest
import scipy.sparse as sp

import lgh_b200 as L

from test_gpu_strip_tiles import _banded, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,n,w", [(2, 21401, 64), (2, 21401, 65), (2, 21401, 67),
                                   (2, 6001, 219), (2, 4001, 502),
                                   (4, 43001, 48), (4, 43001, 51),
                                   (4, 12001, 219)])
def test_four_packs(cuda_device, R, n, w):
    A = _banded(n, n + w)
    X = np.random.default_rng(w).standard_normal((n, w))
    _check(A, X, False, R)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("w", [9, 60, 221])
def test_diagonal(cuda_device, fp32, w):
    n = 21401
    A = sp.diags(np.random.default_rng(w).standard_normal(n)).tocsr()
    X = np.random.default_rng(w + 1).standard_normal((n, w))
    csr = dict(n=n, rowptr=A.indptr.astype(np.int64),
               colidx=A.indices.astype(np.int32), vals=A.data)
    Y, used = L.test_spmm_strip(L.Mat(csr), X, fp32=fp32)
    assert used == 2
    # one product with the roundings of the value and of X
    u = 2.0 ** (-24 if fp32 else -53)
    assert np.all(np.abs(Y - A @ X) <= 4 * u * np.abs(A @ X))
