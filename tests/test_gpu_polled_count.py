"""The active-column count of a solve reaches the host through a pinned slot
that it polls, or, when the process has handed out all of them (64), by a
copy: more workspaces than slots, whose solves must give the same bits and
take the same iterations either way, and again after some were given back."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


def test_more_workspaces_than_slots(cuda_device):
    side = 50                               # two levels
    mass = P.lumped_mass(side, 2)
    Z = L.Mat(P.z_operator(side, 2, 25.0, mass))
    X = np.random.default_rng(1).standard_normal((side * side, 70))
    priors, first = [], None

    def more(count):
        for _ in range(count):
            p = L.Prior(Z=Z, mass=mass)
            got = (p.solve_block(X), p.solve(X[:, 3]))
            priors.append(p)
            yield got + (p.info()["mean_col_iters"],)

    # a block and a vector workspace each: 80 slots asked for
    for got in list(more(40)):
        first = first or got
        assert np.array_equal(got[0], first[0])
        assert np.array_equal(got[1], first[1])
        assert got[2] == first[2]
    del priors[::2]
    for got in list(more(10)):
        assert np.array_equal(got[0], first[0])
        assert np.array_equal(got[1], first[1])
        assert got[2] == first[2]
