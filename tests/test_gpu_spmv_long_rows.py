"""The single-vector product where a few rows hold many times the mean
length: at the row lengths where the shape for such operators changes (48
entries a round, up to 16 rounds).  Bound as in test_gpu_spmv_shapes.py: at
most 800 products in any order, 800 u |A| |x| = 9e-14."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [2, 30, 48])
@pytest.mark.parametrize("long", [384, 385, 768, 769, 800])
def test_long_rows(cuda_device, mean, long):
    n = 30001
    rng = np.random.default_rng(long + mean)
    cnt = np.full(n, mean - 1)
    cnt[::500] = long
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    row = np.repeat(np.arange(n), cnt)
    ci = ((row + 37 * (np.arange(rp[-1]) - rp[row])) % n).astype(np.int32)
    A = dict(n=n, rowptr=rp, colidx=ci, vals=rng.standard_normal(rp[-1]))
    x = rng.standard_normal(n)
    y = L.Mat(A).mult(x)
    mag = P.csr_matvec(dict(A, vals=np.abs(A["vals"])), np.abs(x))
    assert np.all(np.abs(y - P.csr_matvec(A, x)) <= 9e-14 * mag)
