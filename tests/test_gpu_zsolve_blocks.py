"""Blocked multigrid-PCG Z-solves against a sparse direct solve, at the
widths where the block passes change form: one vector (unaligned source and
result), the last width whose column sums the last CTA adds (32) and the
first that a launch of its own adds, the edges of the packs per thread, a
width past the 512 columns of one tile.  A zero column stays exactly zero
and changes nothing for the others.

Tolerances: the solves stop at a preconditioned residual of 1e-12, and the
preconditioned operator's condition number is below 10, so the solution is
good to a few 1e-11; 1e-9 leaves the rounding of an operator of condition
1e3.  FP32 blocks round the data and the result to 6e-8, amplified at most
as much as the data itself: 1e-5."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu

CASES = {
    "2d": lambda: P.z_operator(61, 2, 25.0, P.lumped_mass(61, 2)),
    "3d": lambda: P.z_operator(17, 3, 16.0, P.lumped_mass(17, 3)),
}


@pytest.fixture(scope="module")
def problems(cuda_device):
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl
    out = {}
    for k, f in CASES.items():
        Z = f()
        n = Z["n"]
        A = sp.csc_matrix(sp.csr_matrix((Z["vals"], Z["colidx"], Z["rowptr"]),
                                        shape=(n, n)))
        X = np.random.default_rng(8).standard_normal((n, 520))
        X[:, 2] = 0.0
        out[k] = (L.Prior(Z=L.Mat(Z), mass=np.ones(n)), X,
                  sl.splu(A).solve(X))
    return out


@pytest.mark.parametrize("w", [1, 3, 4, 5, 8, 31, 32, 33, 64, 66, 131, 220,
                               256, 520])
@pytest.mark.parametrize("name", sorted(CASES))
def test_block_solve(problems, name, w):
    prior, X, ref = problems[name]
    Y = prior.solve_block(X[:, :w])
    nrm = np.linalg.norm(ref[:, :w], axis=0)
    nrm[2:3] = 1.0
    assert np.max(np.linalg.norm(Y - ref[:, :w], axis=0) / nrm) < 1e-9
    if w > 2:
        assert not Y[:, 2].any()
    if w == 1:
        y = prior.solve(X[:, 0])
        assert np.linalg.norm(y - ref[:, 0]) < 1e-9 * nrm[0]


@pytest.mark.parametrize("w", [1, 7, 33, 130, 260])
@pytest.mark.parametrize("name", sorted(CASES))
def test_block_solve_fp32(problems, name, w):
    prior, X, ref = problems[name]
    Y = L.test_zsolve(prior, X[:, :w], fp32=True)
    nrm = np.linalg.norm(ref[:, :w], axis=0)
    nrm[2:3] = 1.0
    assert np.max(np.linalg.norm(Y - ref[:, :w], axis=0) / nrm) < 1e-5


@pytest.mark.parametrize("w", [1, 4, 9, 17, 64, 65, 130])
@pytest.mark.parametrize("n", [40, 333, 1490])
def test_coarse_only(cuda_device, n, w):
    """A prior of one level: the V-cycle is the dense coarse solve."""
    rng = np.random.default_rng(n)
    d = 2.0 + rng.random(n)
    e = -0.4 - 0.5 * rng.random(n - 1)
    i = np.arange(n)
    Z = P.coo_to_csr(n, np.concatenate([i, i[1:], i[:-1]]),
                     np.concatenate([i, i[:-1], i[1:]]),
                     np.concatenate([d, e, e]))
    A = P.csr_to_dense(Z)
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(n))
    X = rng.standard_normal((n, w))
    ref = np.linalg.solve(A, X)
    # FP64: condition below 100 and n terms; FP32 in and out: 6e-8
    Y, smax = L.test_vcycle(prior, X)
    assert len(smax) == 1
    assert np.linalg.norm(Y - ref) < 1e-11 * np.linalg.norm(ref)
    Y, _ = L.test_vcycle(prior, X, fp32=True)
    assert np.linalg.norm(Y - ref) < 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("w", [1, 3, 5, 33, 66, 131])
@pytest.mark.parametrize("rtol", [0.5, 1e-2, 1e-6])
@pytest.mark.parametrize("mode", [2, 3])
def test_fixed_count(problems, mode, rtol, w):
    """The fixed-count iteration, from two steps (the first and the last
    step's own forms) to a dozen, against its steps x += b_k z, r -= b_k Z z
    in numpy around the library's V-cycle, b_k the Chebyshev recurrence's
    step lengths.  Rounding only: 1e-12."""
    _, X, _ = problems["2d"]
    Z = CASES["2d"]()
    X = X[:, :w]
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(Z["n"]),
                    opts=L.prior_opts(blocked_mode=mode, cheb_rtol=rtol))
    info = prior.info()
    lo, hi, nit = info["lmin"], info["lmax"], info["nit"]
    A = P.csr_to_dense(Z)
    theta, delta = 0.5 * (hi + lo), 0.5 * (hi - lo)
    s1 = theta / delta
    b, rho = 1.0 / theta, 1.0 / s1
    x, r = np.zeros_like(X), X.copy()
    for k in range(nit):
        if k > 0:
            rho = 1.0 / (2.0 * s1 - rho)
            b = 2.0 * rho / delta
        z = L.test_vcycle(prior, r)[0]
        x, r = x + b * z, r - b * (A @ z)
    Y = prior.solve_block(X)
    assert np.linalg.norm(Y - x) < 1e-12 * np.linalg.norm(x)
