"""Performance cases of the GLR + prior path on one B200.

Every case is one call, or one short sequence of calls, that a program using
the library makes on resident data: device CSR operators for B and Z, a prior
with its preconditioner, and, where the call needs one, a finished GLR object.
Blocks are column-major FP64 device arrays, as the C ABI takes them; the
request loop's blocks are host arrays.

The data are those of the benchmark configurations (lgh_b200/problems.py) on
a grid of any shape, with the amplitude field, the shift and the right-hand
sides drawn from the seed: grid points on the unit square or cube, lumped
mass, Z = h^(d-2) L + s M (L the Neumann graph Laplacian, 5- or 7-point), and
B a Gaussian x Wendland-C2 kernel matrix.  The kernel's length and radius are
given in grid steps, at the ratios of the configurations (512^2: 2.56 and
7.67 steps, 183 entries per row; 96^3 and 128^3: 1.14-1.27 and 2.4-2.5 steps,
57-81 per row).

Kinds of case:
  job     one GLR build, a blocked solve and a logdet (the benchmark's job)
  extend  a build, then an incremental extension of it
  zsolve  the prior's blocked Z-solve, multigrid PCG or fixed-count Chebyshev
  zvec    the prior's single-vector Z-solve
  solve, sample, factor, filter, apply
          the single-vector operations with H(c) = B + c R
  batch   many right-hand sides at many shifts, solved or sampled
  serve   a burst of requests through the request loop
"""

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "lgpsf-hessian_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lgh_b200 as L  # noqa: E402

F64 = torch.float64


# --------------------------------------------------------------------------
# the cases


def listed():
    return [
        # the headline: a 512^2 build at rank 200 + 20, 16 right-hand sides
        dict(name="job_2d", kind="job", nx=512, ny=512, nz=1, ell=220,
             rank=200, q=1, prec="fp64", m=16),
        # the same job in mixed precision on a ragged grid and sketch
        dict(name="job_2d_mixed_ragged", kind="job", nx=389, ny=511, nz=1,
             ell=131, rank=117, q=1, prec="mixed", m=7),
        # a small build: an inner step of an outer loop, bound by latency
        dict(name="job_small", kind="job", nx=64, ny=64, nz=1, ell=60,
             rank=50, q=1, prec="fp64", m=4),
        # a 3D build that turns out too small and is widened
        dict(name="extend_3d_mixed", kind="extend", nx=67, ny=64, nz=61,
             ell=90, k=70, q=1, prec="mixed"),
        # blocked prior solves (prior samples, preconditioned directions)
        dict(name="zsolve_3d_w33", kind="zsolve", nx=96, ny=96, nz=96, w=33,
             mode=0, rtol=1e-10),
        dict(name="zsolve_2d_cheb_w48", kind="zsolve", nx=257, ny=255, nz=1,
             w=48, mode=2, rtol=1e-10),
        # the smallest call: one vector on a 64^2 grid
        dict(name="zvec_small", kind="zvec", nx=64, ny=64, nz=1, rtol=1e-12),
        # one right-hand side: a Newton step
        dict(name="solve_vec", kind="solve", nx=512, ny=512, nz=1, ell=220,
             rank=200, c=1.0),
        # hyperparameter sweeps: samples and solves at many shifts
        dict(name="sample_batch", kind="batch", op="sample", nx=512, ny=512,
             nz=1, ell=220, rank=200, prec="fp64", nshift=16, m=96),
        dict(name="solve_batch_mixed", kind="batch", op="solve", nx=64, ny=64,
             nz=64, ell=165, rank=150, prec="mixed", nshift=8, m=61),
        # one exact Hessian action: a Krylov or a check step
        dict(name="apply_vec", kind="apply", nx=512, ny=512, nz=1, ell=60,
             rank=50, c=0.3),
        # a burst of independent requests against a resident object
        dict(name="serve_burst", kind="serve", nx=512, ny=512, nz=1, ell=220,
             rank=200, prec="mixed", requests=6, mmax=32),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "extend", "zsolve", "zsolve", "zvec",
                       "solve", "sample", "factor", "filter", "batch",
                       "batch", "apply", "serve"])
    if rng.random() < 0.6:
        nx, ny, nz = _logu(rng, 48, 512), _logu(rng, 48, 512), 1
    else:
        nx, ny, nz = (_logu(rng, 16, 64) for _ in range(3))
    ell = _logu(rng, 24, 220)
    rank = max(8, ell - max(4, ell // rng.choice([8, 11, 16])))
    prec = rng.choice(["fp64", "mixed"])
    c = round(math.exp(rng.uniform(math.log(1e-2), math.log(1e2))), 4)
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "job":
        case.update(ell=ell, rank=rank, q=rng.choice([0, 1]), prec=prec,
                    m=_logu(rng, 1, 16))
    elif kind == "extend":
        half = _logu(rng, 16, 100)
        case.update(ell=half, k=_logu(rng, 5, half), q=1, prec=prec)
    elif kind == "zsolve":
        case.update(w=_logu(rng, 1, 128), mode=rng.choice([0, 0, 2, 3]),
                    rtol=rng.choice([1e-8, 1e-10, 1e-12]))
    elif kind == "zvec":
        case.update(rtol=rng.choice([1e-8, 1e-10, 1e-12]))
    elif kind in ("solve", "sample", "factor", "filter", "apply"):
        case.update(ell=ell, rank=rank, c=c)
    elif kind == "batch":
        case.update(op=rng.choice(["solve", "sample"]), ell=ell, rank=rank,
                    prec=prec, nshift=_logu(rng, 1, 16), m=_logu(rng, 2, 96))
    else:
        case.update(ell=ell, rank=rank, prec=prec,
                    requests=rng.randint(2, 6), mmax=_logu(rng, 2, 32))
    return case


# --------------------------------------------------------------------------
# operators


class _Grid:
    """Mass, Z and B of a grid case, on the GPU, from the seed."""

    def __init__(self, case, seed):
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        self.dim = 2 if self.nz == 1 else 3
        self.n = self.nx * self.ny * self.nz
        g = np.random.default_rng(1000003 * int(seed) + 17)
        self.phase = g.uniform(0.0, 2.0 * np.pi, 3)
        base = 25.0 if self.dim == 2 else 16.0
        self.shift = base * g.uniform(0.9, 1.1)
        self.h = 1.0 / (max(self.nx, self.ny, self.nz) - 1)
        if self.dim == 2:
            self.lb, self.rho = 2.56, 7.67
        else:
            self.lb, self.rho = 1.2, 2.45
        dev = torch.device("cuda")
        i = torch.arange(self.n, device=dev)
        self.c = [i % self.nx, (i // self.nx) % self.ny,
                  i // (self.nx * self.ny)]
        self.dims = [self.nx, self.ny, self.nz]
        m = torch.full((self.n,), self.h ** self.dim, dtype=F64, device=dev)
        for d in range(self.dim):
            edge = (self.c[d] == 0) | (self.c[d] == self.dims[d] - 1)
            m = torch.where(edge, 0.5 * m, m)
        self.mass = m
        x = [self.c[d].to(F64) / (self.dims[d] - 1) for d in range(self.dim)]
        t = [2 * np.pi * x[d] + self.phase[d] for d in range(self.dim)]
        a = 0.5 * torch.sin(t[0])
        a = a * (torch.cos(t[1]) if self.dim == 2
                 else torch.sin(t[1]) * torch.sin(t[2]))
        self.a = 1.0 + a

    def _entries(self, offs, value):
        """(inside, column, value) of every row at each grid offset, the
        offsets in ascending column order; outside the grid the column is
        the row itself."""
        i = torch.arange(self.n, device=self.mass.device)
        for dz, dy, dx in sorted(offs):
            ok = (self.c[0] + dx >= 0) & (self.c[0] + dx < self.nx) \
                & (self.c[1] + dy >= 0) & (self.c[1] + dy < self.ny) \
                & (self.c[2] + dz >= 0) & (self.c[2] + dz < self.nz)
            j = torch.where(ok, i + dx + self.nx * (dy + self.ny * dz), i)
            yield ok, j, value((dz, dy, dx), j)

    def _csr(self, offs, value):
        """CSR arrays (columns ascending) of the entries inside the grid."""
        cols, vals, oks = [], [], []
        for ok, j, v in self._entries(offs, value):
            cols.append(j.to(torch.int32))
            vals.append(v)
            oks.append(ok)
        ok = torch.stack(oks, 1)
        rowptr = torch.zeros(self.n + 1, dtype=torch.int64, device=ok.device)
        torch.cumsum(ok.sum(1), 0, out=rowptr[1:])
        col = torch.stack(cols, 1)[ok]
        val = torch.stack(vals, 1)[ok]
        return rowptr, col.contiguous(), val.contiguous()

    def zstencil(self):
        """(diagonal, off-diagonal value) of Z."""
        deg = torch.zeros(self.n, dtype=F64, device=self.mass.device)
        for d in range(self.dim):
            deg += (self.c[d] > 0).to(F64)
            deg += (self.c[d] < self.dims[d] - 1).to(F64)
        s = self.h ** (self.dim - 2)
        return s * deg + self.shift * self.mass, -s

    def zcsr(self):
        diag, off = self.zstencil()
        offs = [(0, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0)]
        if self.dim == 3:
            offs += [(1, 0, 0), (-1, 0, 0)]
        const = torch.full_like(diag, off)
        return self._csr(offs, lambda o, j: diag if o == (0, 0, 0) else const)

    def _kernel(self):
        """(offsets, value) of B."""
        r = int(math.floor(self.rho))
        rz = r if self.dim == 3 else 0
        offs = [(dz, dy, dx) for dz in range(-rz, rz + 1)
                for dy in range(-r, r + 1) for dx in range(-r, r + 1)
                if dx * dx + dy * dy + dz * dz < self.rho ** 2]
        am = self.a * self.mass

        def value(o, j):
            d = math.sqrt(o[0] ** 2 + o[1] ** 2 + o[2] ** 2)
            t = d / self.rho
            k = math.exp(-d * d / (2 * self.lb ** 2)) * (1 - t) ** 4 * (4 * t + 1)
            return am * am[j] * k

        return offs, value

    def bcsr(self):
        return self._csr(*self._kernel())

    def bmul(self, x):
        """B x of one vector, offset by offset."""
        y = torch.zeros_like(x)
        for ok, j, v in self._entries(*self._kernel()):
            y += torch.where(ok, v * x[j], torch.zeros_like(x))
        return y

    def zmul(self, x, diag, off):
        """Z x of a block x (m, n), from the stencil."""
        v = x.view(-1, self.nz, self.ny, self.nx)
        y = (diag * x).view_as(v)
        for d in range(self.dim):
            k = 3 - d
            if v.shape[k] < 2:
                continue
            n = v.shape[k]
            y.narrow(k, 0, n - 1).add_(v.narrow(k, 1, n - 1), alpha=off)
            y.narrow(k, 1, n - 1).add_(v.narrow(k, 0, n - 1), alpha=off)
        return y.view_as(x)

    def zinv(self, b):
        """Z^{-1} b of a block b (m, n): conjugate gradients to the last
        digits, then refinement steps on the residual."""
        diag, off = self.zstencil()
        x = torch.zeros_like(b)
        for _ in range(3):
            r = b - self.zmul(x, diag, off)
            e = torch.zeros_like(b)
            z = r / diag
            p = z.clone()
            rz = (r * z).sum(1, keepdim=True)
            stop = 1e-20 * rz
            for it in range(20000):
                q = self.zmul(p, diag, off)
                al = rz / (p * q).sum(1, keepdim=True)
                al = torch.where(rz > stop, al, torch.zeros_like(al))
                e += al * p
                r -= al * q
                z = r / diag
                new = (r * z).sum(1, keepdim=True)
                be = torch.where(rz > stop, new / rz, torch.zeros_like(rz))
                p = z + be * p
                rz = torch.where(rz > stop, new, rz)
                if it % 50 == 49 and not bool((rz > stop).any()):
                    break
            x += e
        return x


def _mat(csr):
    """A device CSR Mat from device arrays (copied by the library)."""
    A = L.Mat.__new__(L.Mat)
    A.h = L.P()
    A.n = csr[0].numel() - 1
    torch.cuda.synchronize()
    L._chk(L.load().lgh_mat_create_csr(A.n, csr[0].data_ptr(),
                                       csr[1].data_ptr(), csr[2].data_ptr(),
                                       L.LGH_MEM_DEVICE, ctypes.byref(A.h)),
           "lgh_mat_create_csr")
    return A


def _vec(t):
    """A Vec over a tensor's memory (the tensor is kept by the caller)."""
    v = L.P()
    L._chk(L.load().lgh_vec_create_with_array(t.numel(), t.data_ptr(),
                                              ctypes.byref(v)),
           "lgh_vec_create_with_array")
    return v


def _randn(seed, tag, *shape):
    g = torch.Generator(device="cuda")
    g.manual_seed(7919 * int(seed) + tag)
    return torch.randn(*shape, generator=g, dtype=F64, device="cuda")


# --------------------------------------------------------------------------
# prepare / run


class _State:
    pass


def _glr(s, case):
    opts = L.glr_opts(ell=case["ell"], q_power=case.get("q", 1), seed=0,
                      trunc_rel=0.0, check=1)
    prec = L.PREC_MIXED if case.get("prec") == "mixed" else L.PREC_FP64
    ex = L.exec_opts(rank_cap=case.get("rank", 0), precision=prec)
    return L.Glr(s.B, s.prior, opts, exec=ex)


def _rhs(case, seed, n):
    """The right-hand sides of a case: (columns, n) on the GPU."""
    cols = case.get("m", case.get("w", 1))
    return _randn(seed, 1, cols, n)


def _requests(case, seed):
    """(kind, shift, width) of each request: mostly solves, some samples, a
    logdet now and then; widths spread over 1..mmax, shifts over six
    decades."""
    g = np.random.default_rng(31 * int(seed) + 5)
    kinds = [L.Server.SOLVE, L.Server.SAMPLE, L.Server.SOLVE,
             L.Server.LOGDET, L.Server.SOLVE, L.Server.SAMPLE]
    out = []
    for r in range(case["requests"]):
        m = 1 + (r * 11 + 5) * (case["mmax"] - 1) % case["mmax"]
        out.append((kinds[r % 6], float(10.0 ** g.uniform(-3, 3)), m))
    return out


def prepare(case, seed):
    L.load()
    s = _State()
    s.case, s.kind = case, case["kind"]
    grid = _Grid(case, seed)
    s.n = grid.n
    s.Z = _mat(grid.zcsr())
    po = L.prior_opts(ksp_rtol=case.get("rtol", 1e-10),
                      cheb_rtol=case.get("rtol", 1e-10),
                      blocked_mode=case.get("mode", 0))
    s.prior = L.Prior(Z=s.Z, mass=grid.mass.cpu().numpy(), opts=po)
    if s.kind not in ("zsolve", "zvec"):
        s.B = _mat(grid.bcsr())
    if s.kind not in ("zsolve", "zvec", "job", "extend"):
        s.glr = _glr(s, case)
    if s.kind == "serve":
        s.server = L.Server(s.glr, slots=64)
        s.reqs = []
        for r, (kind, c, m) in enumerate(_requests(case, seed)):
            X = None
            if kind != L.Server.LOGDET:
                X = _randn(seed, 100 + r, m, s.n).cpu().numpy().T
            s.reqs.append((kind, c, X))
        return s
    s.x = _rhs(case, seed, s.n)
    if s.kind == "batch":
        g = np.random.default_rng(13 * int(seed) + 3)
        s.cs = 10.0 ** g.uniform(-2, 2, case["nshift"])
        s.y = torch.empty(case["nshift"] * case["m"], s.n, dtype=F64,
                          device="cuda")
    else:
        s.cs = np.array([case.get("c", 1.0)])
        s.y = torch.empty_like(s.x)
    s.vx, s.vy = _vec(s.x), _vec(s.y)
    if s.kind == "filter":
        s.flam = np.sqrt(np.abs(s.glr.eigs()) + case["c"])
    torch.cuda.synchronize()
    return s


def run(s):
    lib, case, kind = L.load(), s.case, s.kind
    if kind == "job":
        s.glr = None            # the previous job's object is released first
        s.glr = g = _glr(s, case)
        L._chk(lib.lgh_glr_solve_batch(g.h, 1, s.cs.ctypes.data_as(L.c_dbl_p),
                                       case["m"], s.x.data_ptr(), s.n,
                                       s.y.data_ptr(), s.n),
               "lgh_glr_solve_batch")
        return g.eigs(), s.y, g.logdet(float(s.cs[0]))
    if kind == "extend":
        s.glr = None
        s.glr = g = _glr(s, case)
        first = g.eigs()
        g.extend(case["k"])
        L._chk(lib.lgh_glr_sample(g.h, 1.0, s.vx, s.vy), "lgh_glr_sample")
        return first, g.eigs(), s.y
    if kind == "zsolve":
        L._chk(lib.lgh_prior_solve_block(s.prior.h, case["w"], s.x.data_ptr(),
                                         s.n, s.y.data_ptr(), s.n),
               "lgh_prior_solve_block")
        return s.y
    if kind == "zvec":
        L._chk(lib.lgh_prior_solve(s.prior.h, s.vx, s.vy), "lgh_prior_solve")
        return s.y
    if kind == "batch":
        f = lib.lgh_glr_solve_batch if case["op"] == "solve" \
            else lib.lgh_glr_sample_batch
        L._chk(f(s.glr.h, case["nshift"], s.cs.ctypes.data_as(L.c_dbl_p),
                 case["m"], s.x.data_ptr(), s.n, s.y.data_ptr(), s.n),
               "lgh_glr_%s_batch" % case["op"])
        return s.y
    if kind == "serve":
        ids = [s.server.submit(k, c, X) for k, c, X in s.reqs]
        return [s.server.wait(i)[0] for i in ids]
    c = float(s.cs[0])
    if kind == "solve":
        rc = lib.lgh_glr_solve(s.glr.h, c, s.vx, s.vy)
    elif kind == "sample":
        rc = lib.lgh_glr_sample(s.glr.h, c, s.vx, s.vy)
    elif kind == "factor":
        rc = lib.lgh_glr_factor(s.glr.h, c, 0, s.vx, s.vy)
    elif kind == "filter":
        rc = lib.lgh_glr_filter(s.glr.h, s.flam.ctypes.data_as(L.c_dbl_p),
                                math.sqrt(c), s.vx, s.vy)
    else:
        rc = lib.lgh_glr_apply(s.glr.h, c, s.vx, s.vy)
    L._chk(rc, "lgh_glr_" + kind)
    return s.y


# --------------------------------------------------------------------------
# work / exact


def _counts(case):
    """(n, entries of Z, entries of B), interior stencils everywhere."""
    n = case["nx"] * case["ny"] * case["nz"]
    two = case["nz"] == 1
    return n, n * (5 if two else 7), n * (185 if two else 57)


def work(case):
    """What one pass cannot do without: operators, the object's basis and
    the blocks once each (8 bytes a value, 4 an index), one product with Z
    per Z-solve, and the dense products."""
    n, nz, nb = _counts(case)
    kind = case["kind"]
    zb, bb = 12.0 * nz, 12.0 * nb
    if kind in ("job", "extend"):
        ell = case["ell"] + case.get("k", 0)
        rank = case.get("rank", ell)
        m = case.get("m", 1)
        napp = case["q"] + 2
        north = 2 * (case["q"] + 1)
        flops = napp * ell * (2.0 * nb + 4.0 * nz) + 4.0 * m * nz
        flops += n * ell * (2.0 * north * ell + 2.0 * ell + 4.0 * rank)
        es = 4 if case["prec"] == "mixed" else 8
        by = zb + bb + 8.0 * n + es * n * rank + 16.0 * n * m
        return dict(bytes=by, flops=flops)
    if kind in ("zsolve", "zvec"):
        w = case.get("w", 1)
        return dict(bytes=zb + 16.0 * n * w, flops=2.0 * nz * w)
    rank = case["rank"]
    ub = 8.0 * n * rank
    if kind == "batch":
        m, ns = case["m"], case["nshift"]
        solves = 2 if case["op"] == "solve" else 1
        return dict(bytes=zb + 2 * ub + 8.0 * n * m * (1 + ns),
                    flops=2.0 * nz * m * solves
                    + 2.0 * n * rank * m * (1 + ns))
    if kind == "serve":
        m = 0.5 * (1 + case["mmax"]) * case["requests"]
        return dict(bytes=zb + 2 * ub + 16.0 * n * m,
                    flops=4.0 * nz * m + 4.0 * n * rank * m)
    if kind == "apply":
        return dict(bytes=bb + zb + 24.0 * n, flops=2.0 * nb + 4.0 * nz)
    if kind == "filter":
        return dict(bytes=ub + 16.0 * n, flops=4.0 * n * rank)
    return dict(bytes=zb + ub + 16.0 * n, flops=4.0 * nz + 4.0 * n * rank)


def exact(case, seed):
    """The Z-solves and the Hessian action in 64 bits, without the library;
    the other kinds depend on a randomized low-rank model and have none."""
    kind = case["kind"]
    if kind not in ("zsolve", "zvec", "apply"):
        return None
    grid = _Grid(case, seed)
    x = _rhs(case, seed, grid.n)
    if kind in ("zsolve", "zvec"):
        return grid.zinv(x)
    diag, off = grid.zstencil()
    y = grid.bmul(x[0]).reshape(1, -1)
    r = grid.zmul(grid.zmul(x, diag, off) / grid.mass, diag, off)
    return y + case["c"] * r
