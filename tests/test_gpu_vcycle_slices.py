"""An operator whose neighbour band does not fit the smoothers' L2 budget is
swept in column slices by the V-cycle's passes: the budget forced down to
one pack a slice, to a few packs, and slicing off.  The slices give the
values of one sweep; only the packs per thread differ, which changes no
column's arithmetic, so they are the same bits."""

import numpy as np
import pytest

import lgh_b200 as L
import lgh_b200.problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [3, 67, 219])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("dim,side", [(2, 90), (3, 20)])
def test_slices_same_bits(cuda_device, monkeypatch, dim, side, fp32, w):
    mass = P.lumped_mass(side, dim)
    Z = P.z_operator(side, dim, 25.0, mass)
    prior = L.Prior(Z=L.Mat(Z), mass=mass)
    X = np.random.default_rng(w).standard_normal((Z["n"], w))
    out, launches = [], []
    # megabytes; a band is 2 x 90 or 2 x 400 rows of up to 1760 bytes
    for mb in ("0", "0.02", "1e-6"):
        monkeypatch.setenv("LGH_CHEB_L2MB", mb)
        c0 = L.runtime_counters()["launches"]
        out.append(L.test_vcycle(prior, X, fp32)[0])
        launches.append(L.runtime_counters()["launches"] - c0)
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])
    if w > 4:                       # the slices were really taken
        assert launches[0] < launches[1] < launches[2]
