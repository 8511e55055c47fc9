"""Performance cases: what users of the solver run, as one call each.

A case names a matrix family and its grid, the factor's precision and decomposition, the number of
right-hand sides and how the solver is called (``mode``):

* ``step``  new values on a kept analysis, everything on the device: DistributeMatrixDevice,
  Factorize, SolveDevice.  A time step, a Newton step, a serving factor+solve request.
* ``solve`` more right-hand sides against a factor that the program keeps: SolveDevice.
* ``host``  the drop-in sequence of run_sympack2D on host buffers: DistributeMatrix, Factorize,
  Solve, GetSolution.

Families: 2D 5-point and 3D 7-point Laplacians, the 27-point stencil with random couplings, the
quasi-definite 27-point grid (LDL^T), and block-diagonal batches of uneven systems.  Grids come
from the benchmark, the serving ladder and the batching workload; values and right-hand sides come
from the seed, the structure from the case.
"""
import math

import numpy as np
import torch

from sympack_b200 import DistSparseMatrix, generators as G, symPACKMatrix2D, symPACKOptions

SHIFT = 1e-3  # diagonal shift of the 3D Laplacians


def _case(name, family, grid, mode, nrhs=1, precision="FP64", decomposition="LL", ordering="MMD", delta=1e-2):
    nx, ny, nz = (tuple(grid) + (1, 1))[:3]
    c = dict(name=name, family=family, nx=nx, ny=ny, nz=nz, mode=mode, nrhs=nrhs, precision=precision,
             decomposition=decomposition, ordering=ordering, delta=delta)
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # the plain method: run_sympack2D's sequence on a 64 x 64 grid, host buffers; launches and copies count
        _case("dropin_lap2d_64", "lap2d", (64, 64), "host"),
        # the smallest call: one more right-hand side against a small kept factor
        _case("solve1_st27_17", "st27", (17, 17, 17), "solve"),
        # a serving factor+solve request on a 2D grid: many small supernodes, refinement steps
        _case("step_lap2d_362_ir", "lap2d", (362, 362), "step", nrhs=16, precision="FP32_IR"),
        # a large ragged 2D grid, AMD ordering, a few right-hand sides: latency of a deep tree of small panels
        _case("step_lap2d_463_amd", "lap2d", (463, 467), "step", nrhs=3, ordering="AMD"),
        # the headline: 60^3 Laplacian, new values, factor and solve
        _case("step_lap3d_60", "lap3d", (60, 60, 60), "step"),
        # the headline's solve-only calls: time steps with a constant matrix
        _case("solve1_lap3d_60", "lap3d", (60, 60, 60), "solve"),
        _case("solve16_lap3d_60", "lap3d", (60, 60, 60), "solve", nrhs=16),
        # a serving solve-only request: cached FP32 factor, many right-hand sides, refined
        _case("solve50_st27_36_ir", "st27", (36, 36, 36), "solve", nrhs=50, precision="FP32_IR"),
        # large fronts in FP64, the serving ladder's largest grid
        _case("step_st27_60", "st27", (60, 60, 60), "step"),
        # the precision form: 80^3, FP32 factor and refinement
        _case("step_st27_80_ir", "st27", (80, 80, 80), "step", precision="FP32_IR"),
        # symmetric indefinite: LDL^T on the benchmark's quasi-definite grid
        _case("step_qd27_50_ldl", "qd27", (50, 50, 50), "step", decomposition="LDL"),
        # the batching form: 64 uneven systems (nx: how many, ny: the largest n) in one handle
        _case("batch_64", "batch", (64, 20000), "step"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    nrhs = rng.choice([1, 1, rng.randint(2, 16), rng.randint(17, 64)])
    ordering = rng.choice(["MMD", "MMD", "AMD"])
    what = rng.choice(["host", "solve", "solve", "solve_ir", "step2", "step3", "step27", "ir", "ir", "ldl", "batch"])
    near = lambda k: tuple(max(2, k + rng.randint(-3, 3)) for _ in range(3))  # noqa: E731
    if what == "host":
        k = _log(rng, 30, 400)
        return _case(None, "lap2d", (k, k + rng.randint(-3, 3)), "host", nrhs=rng.randint(1, 4), ordering=ordering)
    if what == "solve":
        if rng.random() < 0.5:
            return _case(None, "lap3d", near(_log(rng, 10, 56)), "solve", nrhs, ordering=ordering)
        return _case(None, "st27", near(_log(rng, 10, 48)), "solve", nrhs)
    if what == "solve_ir":
        return _case(None, "st27", near(_log(rng, 10, 48)), "solve", nrhs, "FP32_IR")
    if what == "step2":
        k = _log(rng, 30, 460)
        return _case(None, "lap2d", (k, k + rng.randint(-5, 5)), "step", nrhs, rng.choice(["FP64", "FP32_IR"]), ordering=ordering)
    if what == "step3":
        return _case(None, "lap3d", near(_log(rng, 10, 56)), "step", nrhs, ordering=ordering)
    if what == "step27":
        return _case(None, "st27", near(_log(rng, 10, 54)), "step", nrhs)
    if what == "ir":
        return _case(None, "st27", near(_log(rng, 10, 64)), "step", rng.choice([1, nrhs]), "FP32_IR", delta=rng.choice([1e-2, 1e-5]))
    if what == "ldl":
        return _case(None, "qd27", near(_log(rng, 10, 44)), "step", nrhs, decomposition="LDL")
    return _case(None, "batch", (rng.randint(5, 50), _log(rng, 1000, 6000)), "step", 1, rng.choice(["FP64", "FP32_IR"]))


# ---- structures, analysed once: a program reuses a pattern with new values -----------------------

_kept = {}


class _Structure:
    """The lower triangle's pattern, which entries are diagonal, the systems of a batch, the analysis."""

    def __init__(self, c):
        g = (c["nx"], c["ny"], c["nz"])
        self.offsets = self.shift = None
        if c["family"] == "lap2d":
            a = G.laplacian_2d(g[0], g[1])
        elif c["family"] == "lap3d":
            a = G.laplacian_3d(*g, SHIFT)
        elif c["family"] == "batch":
            systems = G.batch_systems(g[0], 500, g[1], seed=0)
            a = G.block_diagonal(systems)
            self.offsets = a[4]
        else:
            a = G.stencil27(*g, 0.01, 0)  # the quasi-definite grid has the same pattern
        self.n, self.colptr, self.rowind, self.base = a[:4]
        self.cols = np.repeat(np.arange(self.n), np.diff(self.colptr))
        self.rows = self.rowind.astype(np.int64) - 1
        self.diag = self.rows == self.cols
        self.analysis = symPACKMatrix2D()
        self.analysis.Init(_options(c, -1))  # on the host, shared by the handles of every state
        A = DistSparseMatrix.from_lower_csc(self.n, self.colptr, self.rowind, self.base)
        if self.offsets is None:
            self.analysis.SymbolicFactorization(A)
        else:
            self.analysis.SymbolicFactorizationBatch(A, self.offsets)

    def _abs_row_sums(self, keep, mag):
        return np.bincount(self.rows[keep], mag, self.n) + np.bincount(self.cols[keep], mag, self.n)

    def values(self, c, seed):
        rng = np.random.default_rng(seed)
        off, v = ~self.diag, self.base.copy()
        if c["family"] in ("lap2d", "lap3d"):  # the implicit step's shift changes from step to step
            v[self.diag] += SHIFT * rng.uniform()
            return v
        mag = 1.0 - rng.uniform(0.0, 1.0, size=int(off.sum()))  # (0, 1]
        if c["family"] == "st27":
            v[off] = -mag
            v[self.diag] = (1.0 + c["delta"]) * self._abs_row_sums(off, mag)[self.rows[self.diag]]
        elif c["family"] == "qd27":
            i, j = self.cols[off], self.rows[off]
            sign = np.where(rng.uniform(size=self.n) < 0.3, -1.0, 1.0)
            same = sign[i] == sign[j]
            v[off] = np.where(same, -sign[i] * mag, rng.uniform(-1.0, 1.0, size=len(i)))
            s = self._abs_row_sums(np.flatnonzero(off)[same], mag[same])
            v[self.diag] = (sign * np.where(s > 0, s * (1.0 + c["delta"]), 1.0))[self.rows[self.diag]]
        else:  # a batch: Laplacians get a shift each, random graphs new couplings
            o = self.offsets
            graph = np.repeat(np.arange(len(o) - 1) % 2 == 1, np.diff(o))  # odd-numbered systems
            shift = np.repeat(SHIFT * rng.uniform(size=len(o) - 1), np.diff(o))
            ge = graph[self.cols[off]]
            v[off] = np.where(ge, -mag, v[off])
            s = 1.05 * self._abs_row_sums(off, mag)
            s[s == 0] = 1.0
            v[self.diag] = np.where(graph, s, v[self.diag] + shift)[self.rows[self.diag]]
        return v


def _options(c, device):
    return symPACKOptions(device=device, orderingStr=c["ordering"], precision=c["precision"], decomposition=c["decomposition"])


def _structure(c):
    key = tuple(c[k] for k in ("family", "nx", "ny", "nz", "precision", "decomposition", "ordering"))
    if key not in _kept:
        while len(_kept) >= 3:
            _kept.pop(next(iter(_kept)))
        _kept[key] = _Structure(c)
    return _kept[key]


def _rhs(c, n, seed):
    return np.random.default_rng([seed, 1]).standard_normal((c["nrhs"], n))  # column-major n x nrhs


_stream = []


def prepare(case, seed):
    S = _structure(case)
    v, b = S.values(case, seed), _rhs(case, S.n, seed)
    M = symPACKMatrix2D()
    M.Init(_options(case, 0))
    M.SymbolicFactorizationFrom(S.analysis)
    s = {"M": M, "mode": case["mode"], "nrhs": case["nrhs"], "n": S.n}
    if case["mode"] == "host":
        s["A"], s["b"] = DistSparseMatrix.from_lower_csc(S.n, S.colptr, S.rowind, v), np.ascontiguousarray(b).T
        return s
    if not _stream:
        _stream.append(torch.cuda.Stream())
    M.SetStream(_stream[0].cuda_stream)
    s["v"], s["b"] = torch.from_numpy(v).cuda(), torch.from_numpy(b).cuda()
    s["x"] = torch.empty_like(s["b"])
    torch.cuda.synchronize()
    if case["mode"] == "solve":
        M.DistributeMatrixDevice(s["v"].data_ptr())
        M.Factorize()
    return s


def run(s):
    M = s["M"]
    if s["mode"] == "host":
        M.DistributeMatrix(s["A"])
        M.Factorize()
        M.Solve(s["b"])
        return M.GetSolution(nrhs=s["nrhs"])
    if s["mode"] == "step":
        M.DistributeMatrixDevice(s["v"].data_ptr())
        M.Factorize()
    M.SolveDevice(s["b"].data_ptr(), s["x"].data_ptr(), s["nrhs"], s["n"])
    return s["x"]


def work(case):
    """The factor's entries move once when it is written and once in each of the two sweeps of a solve
    (the backward sweep starts when the forward one has ended); A, b and x move once.  The refined form
    cannot reach its backward error without one refinement step: two solves."""
    S = _structure(case)
    inf = S.analysis.info()
    nnz_l = float(np.sum(S.analysis.GetColCounts()[0].astype(np.float64)))
    size, solves = (4, 2) if case["precision"] == "FP32_IR" else (8, 1)
    nbytes = 2 * size * nnz_l * solves + 16.0 * S.n * case["nrhs"]
    flops = 4.0 * nnz_l * case["nrhs"] * solves
    if case["mode"] != "solve":
        nbytes += 8.0 * len(S.rowind) + size * nnz_l
        flops += float(inf.flops_stat)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # FP64: rounding in another order, times the condition of the matrix (1e5 for the largest 2D grid,
    # where x is 7e-14 from exact()).  Refined: any answer of backward error 1e-12 is one, so two of
    # them differ by up to about the condition times that (5e-10 from exact() seen at delta 1e-5).
    if case["precision"] == "FP64":
        return {"rel": 1e-12}
    if case["family"] in ("lap2d", "batch") or case["delta"] < 1e-3:
        return {"rel": 1e-8}
    return {"rel": 1e-10}


def exact(case, seed):
    """x from conjugate gradients in 64 bits, its residual recomputed in extended precision and solved
    for again until the correction is in the last place.  Indefinite A: on the normal equations."""
    S = _structure(case)
    v, b = S.values(case, seed), _rhs(case, S.n, seed)
    n, off = S.n, ~S.diag
    r = np.concatenate([S.rows, S.cols[off]])
    c = np.concatenate([S.cols, S.rows[off]])
    a = np.concatenate([v, v[off]])
    order = np.argsort(r, kind="stable")
    r, c, a = r[order], c[order], a[order]
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=ptr[1:])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.sparse_csr_tensor(torch.from_numpy(ptr), torch.from_numpy(c), torch.from_numpy(a), (n, n)).to(dev)
    d = torch.from_numpy(np.abs(v[S.diag])).to(dev)[:, None]
    indefinite = case["family"] == "qd27"
    scale = 1.0 / (d * d if indefinite else d)

    def solve(rhs):
        res = A @ rhs if indefinite else rhs.clone()
        x = torch.zeros_like(res)
        z = scale * res
        p, rz = z.clone(), (res * z).sum(0)
        stop = 1e-20 * rz
        for it in range(20000):
            q = A @ (A @ p) if indefinite else A @ p
            pq = (p * q).sum(0)
            al = torch.where(pq > 0, rz / torch.where(pq > 0, pq, torch.ones_like(pq)), torch.zeros_like(pq))
            x += al * p
            res -= al * q
            z = scale * res
            new = (res * z).sum(0)
            p = z + torch.where(rz > 0, new / torch.where(rz > 0, rz, torch.ones_like(rz)), torch.zeros_like(rz)) * p
            rz = new
            if it % 20 == 19 and bool((rz <= stop).all()):
                break
        return x

    x = np.zeros((n, case["nrhs"]), np.longdouble)
    al = a.astype(np.longdouble)
    for _ in range(3):
        res = np.empty((n, case["nrhs"]))
        for k in range(case["nrhs"]):
            res[:, k] = (b[k].astype(np.longdouble) - np.add.reduceat(al * x[c, k], ptr[:-1])).astype(np.float64)
        x += solve(torch.from_numpy(res).to(dev)).cpu().numpy()
    x = x.astype(np.float64)
    return x if case["mode"] == "host" else torch.from_numpy(np.ascontiguousarray(x.T))
