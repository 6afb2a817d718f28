"""One block V-cycle on operators whose rows are longer than the merge that
forms the smoothed correction takes (1022 entries): the level keeps A P and
runs the same passes around the corrected residual.  Against the correction
form in numpy, at the widths of tests/test_gpu_vcycle.py's edges and with
its tolerances: each level adds a few roundings of its residuals, FP64
1e-10, FP32 1e-4.  And a solve to 1e-12 against a direct one, 1e-9 (an
operator of condition below 1e5)."""

import numpy as np
import pytest

import lgh_b200 as L

from test_gpu_vcycle import _hierarchy, _vcycle, _wide_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(1700, 511), (1700, 520), (2100, 700)],
                ids=lambda p: "%d_%d" % p)
def problem(request, cuda_device):
    n, half = request.param
    Z = _wide_rows(n, half)
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(n))
    X = np.random.default_rng(6).standard_normal((n, 219))
    smax = L.test_vcycle(prior, X[:, :1])[1]
    levels, Ac = _hierarchy(Z, len(smax))
    return Z, prior, X, _vcycle(levels, Ac, smax, X)


@pytest.mark.parametrize("w", [1, 3, 5, 33, 67, 219])
@pytest.mark.parametrize("fp32", [False, True])
def test_vcycle(problem, fp32, w):
    _, prior, X, ref = problem
    Y = L.test_vcycle(prior, X[:, :w], fp32)[0]
    err = np.linalg.norm(Y - ref[:, :w]) / np.linalg.norm(ref[:, :w])
    assert err < (1e-4 if fp32 else 1e-10), err


def test_solve(problem):
    import scipy.linalg as sl
    Z, prior, X, _ = problem
    n = Z["n"]
    A = np.zeros((n, n))
    A[np.repeat(np.arange(n), np.diff(Z["rowptr"])), Z["colidx"]] = Z["vals"]
    ref = sl.cho_solve(sl.cho_factor(A), X[:, :20])
    Y = prior.solve_block(X[:, :20])
    assert np.linalg.norm(Y - ref) < 1e-9 * np.linalg.norm(ref)
