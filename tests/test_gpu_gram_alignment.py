"""lgh_gram_noalloc on every alignment of its operand: even and odd leading
dimensions, bases on and off a 16-byte boundary, columns at the edges of
fragments (8) and tiles (64), rows at the edges of stages (16) and slices.
The operand's surroundings are NaN, so that a value from outside would show.

n products of two rounded values, summed in any order: n u |X|^T |X|."""

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
@pytest.mark.parametrize("w", [1, 7, 8, 9, 33, 63, 64, 65, 127, 130])
def test_alignments(cuda_device, w, pad, off):
    ld = w + pad
    for n in (1, 15, 17, 129, 300, 1000):
        X = np.random.default_rng(n + w).standard_normal((n, w))
        buf = np.full(off + n * ld + 2, np.nan)
        buf[off:off + n * ld].reshape(n, ld)[:, :w] = X
        dx, dg = L.Vec(data=buf), L.Vec(w * w)
        rc = L.load().lgh_gram_noalloc(n, w, dx.ptr() + 8 * off, ld, dg.ptr(), w)
        assert rc == 0
        G = dg.get().reshape(w, w)
        bound = n * 2.0 ** -53 * (np.abs(X).T @ np.abs(X))
        assert np.all(np.abs(G - X.T @ X) <= 2 * bound + 1e-300), n
        assert np.array_equal(G, G.T)
