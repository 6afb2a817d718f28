"""The dense coarse solve's tiles (k_gemm.cu), alone: a problem below the
coarse size limit has one level, and its V-cycle is the dense solve.  Both
row tiles of narrow blocks (n up to and above 8 rows per SM), the widths
where the tile changes, partial tiles of rows, columns and terms.

The inverse is formed once in FP64, so the result differs from a direct
solve by n u cond (1e3 1e-16 1e3) at most; FP32 blocks round the right-hand
side and the result to 6e-8, the former amplified by up to cond."""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sl

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problems(cuda_device):
    out = {}
    for side in (6, 33, 35, 38):          # n = 36, 1089, 1225, 1444
        Z = P.z_operator(side, 2, 25.0, P.lumped_mass(side, 2))
        n = Z["n"]
        A = sp.csc_matrix(sp.csr_matrix((Z["vals"], Z["colidx"], Z["rowptr"]),
                                        shape=(n, n)))
        X = np.random.default_rng(side).standard_normal((n, 133))
        out[side] = (L.Prior(Z=L.Mat(Z), mass=np.ones(n)), X,
                     sl.splu(A).solve(X))
    return out


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("w", [1, 2, 8, 9, 17, 64, 65, 133])
@pytest.mark.parametrize("side", [6, 33, 35, 38])
def test_dense_coarse(problems, side, w, fp32):
    prior, X, ref = problems[side]
    Y, smax = L.test_vcycle(prior, X[:, :w], fp32)
    assert len(smax) == 1
    err = np.linalg.norm(Y - ref[:, :w], axis=0)
    assert np.max(err / np.linalg.norm(ref[:, :w], axis=0)) < (1e-4 if fp32 else 1e-9)
