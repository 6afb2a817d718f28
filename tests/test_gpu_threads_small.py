"""The small dense kernels from several threads with different sizes: their
shared-memory limit is one per kernel, so a thread with a small matrix must
not lower it between another's opt-in and launch."""

import os
import subprocess
import sys
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


def test_potrf_at_the_optin_sizes(cuda_device):
    """The sizes on both sides of where the opt-in is asked for (40 KB) and of
    the default limit (48 KB): panels of n x 17 doubles, columns of 8 x n
    above 512 rows.  In a process of its own: the limit only ever grows.  The
    factor's residual is within n eps of the norm, and the inverse's within
    n eps cond(L)."""
    code = (
        "import numpy as np, lgh_b200 as L\n"
        "for n in (301, 302, 361, 362, 640, 641, 768, 769):\n"
        "    A = np.random.default_rng(n).standard_normal((n, n))\n"
        "    G = A @ A.T + n * np.eye(n)\n"
        "    F, Li, info = L.test_potrf(G)\n"
        "    assert info[0] == 0, (n, info)\n"
        "    F = np.tril(F); Li = np.tril(Li); eps = n * 2.0 ** -52\n"
        "    assert np.linalg.norm(F @ F.T - G) <= eps * np.linalg.norm(G), n\n"
        "    assert np.linalg.norm(Li @ F - np.eye(n)) <= \\\n"
        "        eps * np.linalg.norm(Li) * np.linalg.norm(F), n\n")
    env = dict(os.environ)
    env["PYTHONPATH"] = os.pathsep.join(
        [os.path.dirname(os.path.dirname(os.path.abspath(L.__file__))),
         env.get("PYTHONPATH", "")])
    p = subprocess.run([sys.executable, "-c", code], env=env, timeout=300,
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-2000:]
