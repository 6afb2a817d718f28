"""The FP64 tensor-core products at the edges of their tiles and copies:
widths around the 8-column fragments and 64-column tiles, row counts that
leave a partial 16-deep stage, leading dimensions of either parity (16- and
8-byte copies), the Gram's upper-triangle form, and the many-shift
combination at odd kept counts.  Reference: numpy products of the same
FP64 values; a sum of n products of unit normals differs by at most a few
sqrt(n) 1e-16 times its terms, so 1e-13 relative to |A| |B| entry by entry
is loose."""

import ctypes

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 255, 4099])
@pytest.mark.parametrize("w", [1, 7, 8, 9, 33, 64, 65, 100, 131, 220])
def test_gram(cuda_device, n, w):
    X = np.random.default_rng(n * 1000 + w).standard_normal((n, w))
    G = L.test_gram(X)
    scale = np.abs(X).T @ np.abs(X)
    assert np.max(np.abs(G - X.T @ X) / scale) < 1e-13
    assert np.array_equal(G, G.T)


@pytest.mark.parametrize("ldx", [70, 71])
def test_gram_unaligned(cuda_device, ldx):
    """lgh_gram_noalloc takes any base and leading dimension."""
    n, w = 513, 69
    buf = np.random.default_rng(2).standard_normal(n * ldx + 1)
    for off in (0, 1):
        X = buf[off:off + n * ldx].reshape(n, ldx)[:, :w]
        v, g = L.Vec(data=buf), L.Vec(w * w)
        L._chk(L.load().lgh_gram_noalloc(
            n, w, ctypes.c_void_p(v.ptr() + 8 * off), ldx,
            ctypes.c_void_p(g.ptr()), w), "lgh_gram_noalloc")
        G = g.get().reshape(w, w)
        assert np.max(np.abs(G - X.T @ X)) < 1e-13 * n


@pytest.mark.parametrize("n,k,m", [(1, 1, 1), (63, 15, 7), (64, 16, 8),
                                   (65, 17, 9), (1000, 131, 65),
                                   (777, 220, 131), (300, 33, 1),
                                   (4097, 60, 50)])
def test_gemm_nn(cuda_device, n, k, m):
    rng = np.random.default_rng(n + k + m)
    X, M = rng.standard_normal((n, k)), rng.standard_normal((k, m))
    Y = L.test_gemm_nn(X, M)
    assert np.max(np.abs(Y - X @ M) / (np.abs(X) @ np.abs(M))) < 1e-13


@pytest.mark.parametrize("rank,m,ns", [(9, 1, 2), (31, 5, 13), (40, 33, 4)])
def test_shift_combination(cuda_device, rank, m, ns):
    """Every shift of a batch against the single-shift call (which combines
    before the second Z-solve): equal to the Z-solves' tolerance."""
    p = P.grid_problem("c1")
    prior = L.Prior(Z=L.Mat(p["Z"]), mass=p["mass"])
    g = L.Glr(L.Mat(p["B"]), prior, L.glr_opts(ell=60, trunc_rel=0.0),
              exec=L.exec_opts(rank_cap=rank))
    R = np.random.default_rng(1).standard_normal((p["N"], m))
    cs = 10.0 ** np.linspace(-2, 2, ns)
    for batch, one in ((g.solve_batch, g.solve), (g.sample_batch, g.sample)):
        out = batch(cs, R)
        for s in (0, ns - 1):
            ref = one(cs[s], R[:, m - 1])
            err = np.linalg.norm(out[s][:, m - 1] - ref)
            assert err < 1e-8 * np.linalg.norm(ref)


@pytest.mark.parametrize("nx,ny,rank", [(40, 31, 5), (64, 64, 50),
                                        (33, 47, 41)])
def test_single_vector_operations(cuda_device, nx, ny, rank):
    """The one-column products U^T x and U w through the filter f(x) = x:
    out = f_c in + U diag(f - f_c) U^T in."""
    n = nx * ny
    rng = np.random.default_rng(rank)
    z = 1.0 + rng.random(n)
    A = rng.standard_normal((n, rank))
    Z = L.Mat(P.diag_csr(z))
    prior = L.Prior(Z=Z, mass=np.ones(n), pc="jacobi")
    g = L.Glr(L.Mat(dense=A @ A.T / n), prior,
              L.glr_opts(ell=rank + 3, trunc_rel=0.0),
              exec=L.exec_opts(rank_cap=rank))
    U, x = g.U(), rng.standard_normal(n)
    f = rng.standard_normal(rank)
    y = g.filter(f, 0.25, x)
    ref = 0.25 * x + U @ ((f - 0.25) * (U.T @ x))
    assert np.linalg.norm(y - ref) < 1e-13 * n ** 0.5 * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [7, 100, 4097])
@pytest.mark.parametrize("nnz", [1, 5, 9, 40, 200])
def test_matvec(cuda_device, n, nnz):
    """The single-vector product at each split of a row, with empty and
    uneven rows."""
    rng = np.random.default_rng(n + nnz)
    cnt = rng.integers(0, 2 * nnz + 1, n)
    cnt[0] = 0
    cnt = np.minimum(cnt, n)
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    ci = np.concatenate([rng.choice(n, c, replace=False) for c in cnt]
                        ).astype(np.int32) if rp[-1] else np.zeros(0, np.int32)
    A = dict(n=n, rowptr=rp, colidx=ci, vals=rng.standard_normal(rp[-1]))
    x = rng.standard_normal(n)
    y = L.Mat(A).mult(x)
    ref = P.csr_matvec(A, x)
    mag = P.csr_matvec(dict(A, vals=np.abs(A["vals"])), np.abs(x))
    assert np.all(np.abs(y - ref) <= 1e-14 * mag + 0.0)
