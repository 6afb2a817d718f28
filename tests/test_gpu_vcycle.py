"""One block V-cycle of the prior's multigrid preconditioner against a numpy
restatement in correction form (two Chebyshev-Jacobi steps from zero,
restriction, coarse solve, prolongation, refreshed residual, two more
steps), on hierarchies rebuilt on the host: the prolongators and Galerkin
operators from lgh_test_mg_galerkin, the smoothing intervals from the
library's lambda_max estimates.

The library forms the same operator in fewer passes, so the two differ by
rounding only: each level adds a few roundings of its residuals and the
coarse solve amplifies them no more than it amplifies the residual itself;
a thousand units in the last place of the result's norm covers both
(FP64 1e-10, which also leaves room for the 1e-13 by which the host's and
the device's prolongators may differ; FP32 1e-4)."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


def _csr(n, A):
    import scipy.sparse as sp
    return sp.csr_matrix((A["vals"], A["colidx"], A["rowptr"]),
                         shape=(n, A.get("m", n)))


def _hierarchy(Z, nlev):
    levels = []
    A = Z
    for _ in range(nlev - 1):
        Pl, Ac = L.test_mg_galerkin(A)
        levels.append((_csr(len(A["rowptr"]) - 1, A),
                       _csr(Pl["n"], Pl)))
        A = Ac
    return levels, _csr(A["n"], A).toarray()


def _vcycle(levels, Ac, smax, r0, l=0):
    if l == len(levels):
        return np.linalg.solve(Ac, r0)
    A, Pl = levels[l]
    di = (1.0 / A.diagonal())[:, None]
    lo, hi = 0.1 * smax[l], 1.1 * smax[l]
    theta, delta = 0.5 * (hi + lo), 0.5 * (hi - lo)
    s1 = theta / delta
    rho = 1.0 / (2.0 * s1 - 1.0 / s1)

    def smooth(x, r):
        d = di * r / theta
        x, r = x + d, r - A @ d
        d = rho / s1 * d + 2.0 * rho / delta * (di * r)
        return x + d, r - A @ d

    x, r = smooth(np.zeros_like(r0), r0)
    x = x + Pl @ _vcycle(levels, Ac, smax, Pl.T @ r, l + 1)
    return smooth(x, r0 - A @ x)[0]


CASES = {
    # two levels, three levels (the second with 30 entries a row and
    # restriction rows of 200), a grid with a row length of 9 on level 1
    "2d": lambda: P.z_operator(45, 2, 25.0, P.lumped_mass(45, 2)),
    "3d": lambda: P.z_operator(26, 3, 16.0, P.lumped_mass(26, 3)),
    "2d_levels": lambda: P.z_operator(130, 2, 25.0, P.lumped_mass(130, 2)),
}


@pytest.fixture(scope="module")
def problems(cuda_device):
    out = {}
    for k, f in CASES.items():
        Z = f()
        m = L.Mat(Z)
        n = Z["n"]
        out[k] = (Z, L.Prior(Z=m, mass=np.ones(n)), {})
    return out


# widths at the edges of the packs per thread (1, 2 or 4 packs: 4 | 5, 64 |
# 65 columns FP64), remainders of each, and a wide block
@pytest.mark.parametrize("w", [1, 3, 5, 9, 33, 64, 67, 130, 219])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_vcycle_matches_correction_form(problems, name, fp32, w):
    Z, prior, memo = problems[name]
    rng = np.random.default_rng(3)
    X = rng.standard_normal((Z["n"], 219))[:, :w]
    Y, smax = L.test_vcycle(prior, X, fp32)
    if "ref" not in memo:
        levels, Ac = _hierarchy(Z, len(smax))
        full = np.random.default_rng(3).standard_normal((Z["n"], 219))
        memo["ref"] = _vcycle(levels, Ac, smax, full)
    ref = memo["ref"][:, :w]
    err = np.linalg.norm(Y - ref) / np.linalg.norm(ref)
    assert err < (1e-4 if fp32 else 1e-10), err


def _wide_rows(n=1700, half=330, seed=4):
    """A banded SPD operator of up to 2 half + 1 entries a row: more lists
    per row than the merge that forms the correction operator keeps in
    registers."""
    i = np.arange(n)
    o = np.arange(-half, half + 1)
    j = i[:, None] + o[None, :]
    ok = (j >= 0) & (j < n)
    w = -np.exp(-np.abs(o) / 60.0)[None, :] * np.ones((n, 1))
    w[:, half] = 0.0
    w = np.where(ok, w, 0.0)
    w[:, half] = -w.sum(1) + 0.05
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int64)
    return dict(n=n, rowptr=rp, colidx=j[ok].astype(np.int32), vals=w[ok])


@pytest.mark.parametrize("half", [20, 120, 330])
def test_vcycle_wide_rows(cuda_device, half):
    Z = _wide_rows(half=half)
    prior = L.Prior(Z=L.Mat(Z), mass=np.ones(Z["n"]))
    X = np.random.default_rng(6).standard_normal((Z["n"], 13))
    Y, smax = L.test_vcycle(prior, X)
    levels, Ac = _hierarchy(Z, len(smax))
    ref = _vcycle(levels, Ac, smax, X)
    assert np.linalg.norm(Y - ref) / np.linalg.norm(ref) < 1e-10
