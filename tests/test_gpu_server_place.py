"""Placement of a request's columns into the request loop's slots, several
per launch (server.cu): more columns than one launch places, a grid whose
size is no multiple of the transposed tile, slots that are not neighbours
(freed by earlier requests), and both kinds of right-hand side; against the
batched operations on the same object."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 1], ids=["fp64", "mixed"])
def glr(request, cuda_device):
    side = 37                               # 1369 rows
    mass = P.lumped_mass(side, 2)
    Z = P.z_operator(side, 2, 25.0, mass)
    n = Z["n"]
    mat = L.Mat(Z)
    prior = L.Prior(Z=mat, mass=mass, opts=L.prior_opts(ksp_rtol=1e-12))
    rng = np.random.default_rng(4)
    B = L.Mat(dense=(lambda A: A @ A.T / n)(rng.standard_normal((n, 20))))
    g = L.Glr(B, prior, L.glr_opts(ell=20, seed=0, check=0),
              exec=L.exec_opts(precision=request.param))
    return n, g, (mat, prior, B)


def _requests(sv, n):
    rng = np.random.default_rng(9)
    # 1 and 33 fill 34 slots, 5 more their neighbours; the 41 of the last are
    # placed as slots come free
    return [(k, 0.5 + j, rng.standard_normal((n, m))) for j, (k, m) in
            enumerate([(sv.SOLVE, 1), (sv.SAMPLE, 33), (sv.SOLVE, 5),
                       (sv.SAMPLE, 3), (sv.SOLVE, 41)])]


def test_columns_of_a_request(glr):
    """A column placed with others, in any slot, gives what it gives as a
    request of its own, bit for bit."""
    n, g, _ = glr
    sv = L.Server(g, slots=48)
    reqs = _requests(sv, n)
    ids = [sv.submit(k, c, X) for k, c, X in reqs]
    outs = [sv.wait(i)[0] for i in ids]
    for (k, c, X), y in zip(reqs, outs):
        for j in range(X.shape[1]):
            one = sv.wait(sv.submit(k, c, X[:, j:j + 1].copy()))[0]
            assert np.array_equal(one[:, 0], y[:, j]), (k, c, j)
    sv.close()


def test_against_batched_operations(glr):
    """FP64: both sides solve to 1e-12 in the preconditioned norm; 1e-8 is
    what the loop's other tests allow between the two.  (A mixed object's
    batched combination rounds to FP32, so there is no such bound for it.)"""
    n, g, _ = glr
    if g.stats()["precision"] != 0:
        return
    sv = L.Server(g, slots=48)
    reqs = _requests(sv, n)
    ids = [sv.submit(k, c, X) for k, c, X in reqs]
    for i, (k, c, X) in zip(ids, reqs):
        y = sv.wait(i)[0]
        ref = (g.solve_batch if k == sv.SOLVE else g.sample_batch)([c], X)[0]
        err = np.linalg.norm(y - ref, axis=0) / np.linalg.norm(ref, axis=0)
        assert np.max(err) < 1e-8, (k, c)
    sv.close()
