"""The small dense kernels from several threads with different sizes: their
shared-memory limit is one per kernel, so a thread with a small matrix must
not lower it between another's opt-in and launch."""

import threading

import numpy as np
import pytest

import lgh_b200 as L

pytestmark = pytest.mark.gpu


def test_potrf_sizes_at_once(cuda_device):
    """Five threads with matrices of a few rows beside three whose panels
    need the opt-in (from n = 362 on)."""
    sizes = (2, 3, 4, 5, 6, 370, 400, 450)
    mats, first, errs = {}, {}, []
    for n in sizes:
        A = np.random.default_rng(n).standard_normal((n, n))
        mats[n] = A @ A.T + n * np.eye(n)
        first[n] = L.test_potrf(mats[n])[0]
    big = [n for n in sizes if n > 360]
    left = len(big)

    def body(n):
        nonlocal left
        try:
            k = 0
            while k < 300 if n in big else left > 0:
                assert np.array_equal(L.test_potrf(mats[n])[0], first[n])
                k += 1
        except Exception as e:              # noqa: BLE001
            errs.append((n, repr(e)))
        if n in big:
            left -= 1

    ts = [threading.Thread(target=body, args=(n,)) for n in sizes]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs, errs
