"""A request's column gives the same bits whatever number of columns is
harvested with it, at sizes where the products U^T r of a wide and a narrow
harvest differ in form: 16 row slices or more (4096 rows), more and fewer
than 8192 coefficients (150 kept: 54 | 55 columns), and more columns than
one 64-column output tile."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("side,slots", [(67, 64), (162, 96)])
def test_width_of_a_harvest(cuda_device, side, slots, prec):
    mass = P.lumped_mass(side, 2)
    Z = L.Mat(P.z_operator(side, 2, 25.0, mass))
    B = L.Mat(P.b_operator(side, 2, 0.02, 4.5 / (side - 1), mass,
                           P.a_field(side, 2, "sincos")))
    prior = L.Prior(Z=Z, mass=mass)
    g = L.Glr(B, prior, L.glr_opts(ell=165, seed=0, trunc_rel=1e-14,
                                    check=0),
              exec=L.exec_opts(precision=prec, rank_cap=150))
    assert g.report["kept"] == 150
    n = side * side
    X = np.random.default_rng(5).standard_normal((n, slots))
    sv = L.Server(g, slots=slots)
    for kind in (sv.SAMPLE, sv.SOLVE):
        wide = sv.wait(sv.submit(kind, 0.7, X))[0]
        for j in range(0, slots, 3):
            one = sv.wait(sv.submit(kind, 0.7, X[:, j:j + 1].copy()))[0]
            assert np.array_equal(one[:, 0], wide[:, j]), (kind, j)
    sv.close()
