"""Fixed-count Z-solves (blocked modes 2 and 3) against direct solves.

The iteration's error is p(V Z) e_0 with V Z self-adjoint in the energy
product <x, Z y>, so the energy norm of the error falls by at most max |p|
over the preconditioned spectrum, which the estimates bracket.  Where lmax /
lmin is above 2.5 the recurrence is Chebyshev's and its count n the smallest
with 2 rho^n <= cheb_rtol: the bound is cheb_rtol.  Below it the steps run
without the direction term: the bound is the maximum of prod |1 - b_k t|,
computed here.  Rounding: 1e-12 in FP64 (a spectrum of 1e4 or less); FP32
blocks round the data and the iterates to 6e-8: 1e-5."""

import math

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


def _anisotropic(side, eps, shift):
    """5-point graph Laplacian with the second direction's weight eps."""
    n = side * side
    i = np.arange(n)
    x, y = i % side, i // side
    rows, cols, vals, d = [], [], [], np.full(n, shift)
    for dx, dy, w in ((1, 0, 1.0), (-1, 0, 1.0), (0, 1, eps), (0, -1, eps)):
        ok = ((x + dx >= 0) & (x + dx < side) & (y + dy >= 0)
              & (y + dy < side))
        rows.append(i[ok])
        cols.append((i + dx + dy * side)[ok])
        vals.append(np.full(ok.sum(), -w))
        d += w * ok
    return P.coo_to_csr(n, np.concatenate(rows + [i]),
                        np.concatenate(cols + [i]), np.concatenate(vals + [d]))


@pytest.fixture(scope="module", params=[1.0, 0.1, 0.03, 0.01])
def problem(request, cuda_device):
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl
    Z = _anisotropic(45, request.param, 0.01)
    A = sp.csc_matrix(sp.csr_matrix((Z["vals"], Z["colidx"], Z["rowptr"]),
                                    shape=(Z["n"], Z["n"])))
    X = np.random.default_rng(8).standard_normal((Z["n"], 131))
    return Z, A, X, sl.splu(A).solve(X)


def _energy(A, E):
    return np.sqrt(np.sum(E * (A @ E), axis=0))


def _bound(info, rtol):
    lo, hi, n = info["lmin"], info["lmax"], info["nit"]
    if hi > 2.5 * lo:
        s = math.sqrt(hi / lo)
        assert 2.0 * ((s - 1.0) / (s + 1.0)) ** n <= rtol
        return rtol
    theta, delta = 0.5 * (hi + lo), 0.5 * (hi - lo)
    t = np.linspace(lo, hi, 4001)
    b, rho = 1.0 / theta, delta / theta
    p = 1.0 - b * t
    for _ in range(1, n):
        rho = 1.0 / (2.0 * theta / delta - rho)
        b = 2.0 * rho / delta
        p = p * (1.0 - b * t)
    return np.max(np.abs(p))


@pytest.mark.parametrize("w", [1, 5, 33, 131])
@pytest.mark.parametrize("rtol", [0.5, 1e-4, 1e-10])
@pytest.mark.parametrize("mode", [2, 3])
def test_error(problem, mode, rtol, w):
    Z, A, X, ref = problem
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(Z["n"]),
                    opts=L.prior_opts(blocked_mode=mode, cheb_rtol=rtol))
    Y = prior.solve_block(X[:, :w])
    err = _energy(A, Y - ref[:, :w]) / _energy(A, ref[:, :w])
    assert np.max(err) <= _bound(prior.info(), rtol) + 1e-12


def test_error_fp32(problem):
    Z, A, X, ref = problem
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(Z["n"]),
                    opts=L.prior_opts(blocked_mode=2, cheb_rtol=1e-6))
    Y = L.test_zsolve(prior, X[:, :33], fp32=True)
    err = _energy(A, Y - ref[:, :33]) / _energy(A, ref[:, :33])
    assert np.max(err) <= _bound(prior.info(), 1e-6) + 1e-5
