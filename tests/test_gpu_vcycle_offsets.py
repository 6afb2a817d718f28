"""The V-cycle's passes with the 64-bit entry offsets that operators of 2^31
entries take give the bits of the 32-bit ones: at every number of packs per
thread, with short rows, rows of hundreds of entries (restriction rows split
over thread groups) and a level that keeps A P."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

from test_gpu_vcycle import _wide_rows

pytestmark = pytest.mark.gpu

CASES = {
    "2d": lambda: P.z_operator(130, 2, 25.0, P.lumped_mass(130, 2)),
    "3d": lambda: P.z_operator(26, 3, 16.0, P.lumped_mass(26, 3)),
    "band": lambda: _wide_rows(1700, 120),
    "wide": lambda: _wide_rows(1700, 520),
}


@pytest.fixture(scope="module")
def priors(cuda_device):
    out = {}
    for k, f in CASES.items():
        Z = f()
        out[k] = (Z["n"], L.Prior(Z=L.Mat(Z), mass=np.ones(Z["n"])))
    return out


@pytest.mark.parametrize("w", [1, 6, 40, 96, 219])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_same_bits(priors, name, fp32, w):
    n, prior = priors[name]
    X = np.random.default_rng(3).standard_normal((n, w))
    Y = L.test_vc_level(prior, X, fp32)
    assert np.all(np.isfinite(Y)) and np.linalg.norm(Y) > 0
    assert np.array_equal(Y, L.test_vc_level(prior, X, fp32, wide=True))
