"""The single-vector product at the edges of the row lengths where its lanes
per row change, with empty rows, and with one long row among short ones.

At most 600 products per row, summed in any order, and the value's and the
vector's own roundings do not enter (both are given): 600 u |A| |x| with u =
1.1e-16, 7e-14."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


def _check(n, cnt, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    ci = np.concatenate([rng.choice(n, c, replace=False) for c in cnt]
                        ).astype(np.int32)
    A = dict(n=n, rowptr=rp, colidx=ci, vals=rng.standard_normal(rp[-1]))
    x = rng.standard_normal(n)
    y = L.Mat(A).mult(x)
    ref = P.csr_matvec(A, x)
    mag = P.csr_matvec(dict(A, vals=np.abs(A["vals"])), np.abs(x))
    assert np.all(np.abs(y - ref) <= 7e-14 * mag)


@pytest.mark.parametrize("nnz", [4, 5, 6, 8, 10, 11, 28, 29, 48, 49, 64, 65, 96,
                                 97, 128, 129, 192, 193, 256, 257, 500])
def test_row_lengths(cuda_device, nnz):
    """Every row of the length, but for an empty one and its neighbour of
    twice as many."""
    n = 1001
    cnt = np.full(n, nnz)
    cnt[n // 2], cnt[n // 2 + 1] = 0, min(2 * nnz, 600)
    _check(n, cnt, nnz)


@pytest.mark.parametrize("long", [39, 41, 79, 81, 225, 385, 600])
def test_long_row_among_short(cuda_device, long):
    n = 777
    cnt = np.full(n, 3)
    cnt[[0, n - 1]] = long, 0
    _check(n, cnt, long)
