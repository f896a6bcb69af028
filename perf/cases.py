"""Timed cases of the library: the calls a program makes, over their size ranges.

A case is a dict of plain values:

  call     spmv | spmm | spmm_f16 | cg | bicgstab | cg_multi | batch | build
  matrix   lap2d | poisson3d | convdiff3d | random_spd | block_dense
  nx ny nz grid of the stencil matrices (lap2d: nz = 1)
  n        rows of random_spd / block_dense
  k        right-hand sides of spmm, spmm_f16, cg_multi
  policy   precision policy of cg, bicgstab, batch
  systems, n_min, n_max  size of a batch (rows log-uniform in [n_min, n_max])

The matrices are the benchmark's families (5-point Laplacian, 7-point Poisson
with row-scaled couplings, upwind convection-diffusion, random diagonally
dominant SPD systems, block-structured matrices), made on the GPU from the
seed.  The solves run to a relative residual far below the usual 1e-10, so
that the solution itself, not only its residual, is determined to about nine
digits: every solve's exact answer is then the x* that its right-hand side was
made from.
"""
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import PKG_DIR, load_package

MF = load_package()
DEV = "cuda"
TOL = {"lap2d": 1e-13, "poisson3d": 1e-13, "convdiff3d": 1e-13, "random_spd": 1e-14}
MAXITER = 20000
MF_ERR_NOT_CONVERGED = 6


# ---------------------------------------------------------------- matrices

class Csr:
    """CSR on the GPU: int32 rowptr and colidx, float64 val."""

    def __init__(self, n, rowptr, colidx, val):
        self.n, self.rowptr, self.colidx, self.val = n, rowptr, colidx, val

    def times(self, x):
        """A x for x of shape (n,) in plain torch, row sums in entry order."""
        return torch.segment_reduce(self.val * x[self.colidx.long()], "sum", offsets=self.rowptr.long(), initial=0.0)


def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _stencil(dims, offsets, coefficient, diagonal):
    """Row-major grid dims (slowest first); offsets are grid vectors in
    ascending column order, the zero vector among them; coefficient(d, i, j)
    gives the entries i -> j of direction d, diagonal(sums of |off|) the rest."""
    n = math.prod(dims)
    i = torch.arange(n, device=DEV)
    at, rest = [], i
    for s in reversed(dims):
        at.insert(0, rest % s)
        rest = rest // s
    stride = [math.prod(dims[d + 1:]) for d in range(len(dims))]
    cols = torch.empty(n, len(offsets), dtype=torch.int64, device=DEV)
    vals = torch.zeros(n, len(offsets), dtype=torch.float64, device=DEV)
    keep = torch.ones(n, len(offsets), dtype=torch.bool, device=DEV)
    for d, o in enumerate(offsets):
        j = i + sum(v * s for v, s in zip(o, stride))
        for a, v, s in zip(at, o, dims):
            keep[:, d] &= (a + v >= 0) & (a + v < s)
        cols[:, d] = j
        if any(o):
            vals[:, d] = torch.where(keep[:, d], coefficient(o, i, j.clamp(0, n - 1)), 0.0)
    vals[:, offsets.index((0,) * len(dims))] = diagonal(vals.abs().sum(1))
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = keep.sum(1).cumsum(0).int()
    return Csr(n, rowptr, cols[keep].int(), vals[keep])


STENCIL2 = [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)]
STENCIL3 = [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0)]


def lap2d(nx, ny):
    return _stencil((ny, nx), STENCIL2, lambda o, i, j: torch.full_like(i, -1, dtype=torch.float64),
                    lambda s: torch.full_like(s, 4.0))


def poisson3d(nx, ny, nz, seed):
    f = 10.0 ** (-3.0 * _uniform(_gen(seed, 2), nx * ny * nz))
    return _stencil((nz, ny, nx), STENCIL3, lambda o, i, j: -(f[i] + f[j]) / 2, lambda s: s + 1e-3)


def convdiff3d(nx, ny, nz, seed):
    """Upwind convection at cell Peclet number 10, the velocity's components
    scaled by up to 10 % from the seed."""
    jitter = (0.9 + 0.1 * _uniform(_gen(seed, 2), 3)).tolist()
    flow = [20.0 * v * t for v, t in zip((0.25, 0.5, 1.0), jitter)]
    upwind = lambda o: -(1.0 + sum(w for v, w in zip(o, flow) if v < 0))  # noqa: E731
    return _stencil((nz, ny, nx), STENCIL3, lambda o, i, j: torch.full_like(i, upwind(o), dtype=torch.float64),
                    lambda s: torch.full_like(s, 6.0 + sum(flow)))


def random_spd(sizes, seed):
    """Random diagonally dominant SPD systems of the given sizes, stacked
    block-diagonally: 8 to 32 draws per row, values N(0, 1) times a row scale
    10^U[-4, 4], symmetrised, diagonal the row's |sum| + 1."""
    g = _gen(seed, 3)
    n = int(sum(sizes))
    size = torch.tensor(sizes, dtype=torch.int64, device=DEV)
    first = torch.repeat_interleave(size.cumsum(0) - size, size)
    own = torch.repeat_interleave(size, size)
    draws = 8 + (25 * _uniform(g, n)).long()
    scale = 10.0 ** (8.0 * _uniform(g, n) - 4.0)
    i = torch.repeat_interleave(torch.arange(n, device=DEV), draws)
    j = first[i] + (_uniform(g, i.numel()) * own[i]).long()
    v = 0.5 * torch.randn(i.numel(), generator=g, device=DEV, dtype=torch.float64) * scale[i]
    off = i != j
    i, j, v = i[off], j[off], v[off]
    d = torch.arange(n, device=DEV)
    key, order = torch.sort(torch.cat([i * n + j, j * n + i, d * (n + 1)]), stable=True)
    v = torch.cat([v, v, torch.zeros(n, dtype=torch.float64, device=DEV)])[order]
    key, count = torch.unique_consecutive(key, return_counts=True)
    v = torch.segment_reduce(v, "sum", lengths=count)
    row, col = key // n, key % n
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.bincount(row, minlength=n).cumsum(0)
    v[row == col] = torch.segment_reduce(v.abs(), "sum", offsets=rowptr) + 1.0
    return Csr(n, rowptr.int(), col.int(), v)


def block_dense(n, seed):
    """Per block row of 16 a dense diagonal block and three dense blocks at
    random block columns (N(0, 1) times 10^U[-2, 2] per block), and four
    random N(0, 1) entries per row; one value per position."""
    g = _gen(seed, 4)
    nb = -(-n // 16)
    b = torch.arange(nb, device=DEV)
    bc = torch.cat([b[:, None], (nb * _uniform(g, nb, 3)).long()], 1)
    t = torch.arange(16, device=DEV)
    r = (16 * b[:, None, None, None] + t[None, None, :, None]).expand(nb, 4, 16, 16)
    c = (16 * bc[:, :, None, None] + t[None, None, None, :]).expand(nb, 4, 16, 16)
    v = torch.randn(nb, 4, 16, 16, generator=g, device=DEV, dtype=torch.float64) * 10.0 ** (
        4.0 * _uniform(g, nb, 4, 1, 1) - 2.0)
    sr = (n * _uniform(g, 4 * n)).long()
    sc = (n * _uniform(g, 4 * n)).long()
    sv = torch.randn(4 * n, generator=g, device=DEV, dtype=torch.float64)
    r, c, v = torch.cat([r.reshape(-1), sr]), torch.cat([c.reshape(-1), sc]), torch.cat([v.reshape(-1), sv])
    keep = (r < n) & (c < n)
    r, c, v = r[keep], c[keep], v[keep]
    key, order = torch.sort(r * n + c, stable=True)
    v = v[order]
    start = torch.ones_like(key, dtype=torch.bool)
    start[1:] = key[1:] != key[:-1]
    key, v = key[start], v[start]
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rowptr[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
    return Csr(n, rowptr.int(), (key % n).int(), v)


def _sizes(case):
    """Rows of a batch's systems: log-uniform, the range's two ends included,
    the same for every seed."""
    lo, hi, m = case["n_min"], case["n_max"], case["systems"]
    u = np.random.RandomState(m).rand(m)
    s = np.rint(lo * (hi / lo) ** u).astype(int)
    s[0], s[-1] = lo, hi
    return s.tolist()


def _matrix(case, seed):
    kind = case["matrix"]
    if kind == "lap2d":
        return lap2d(case["nx"], case["ny"])
    if kind == "poisson3d":
        return poisson3d(case["nx"], case["ny"], case["nz"], seed)
    if kind == "convdiff3d":
        return convdiff3d(case["nx"], case["ny"], case["nz"], seed)
    if kind == "block_dense":
        return block_dense(case["n"], seed)
    return random_spd(_sizes(case) if case["call"] == "batch" else [case["n"]], seed)


def _columns(case, n, seed):
    """The seed's k vectors U[-1, 1], one per row (column-major n x k)."""
    return 2.0 * _uniform(_gen(seed, 1), case.get("k", 1), n) - 1.0


# ------------------------------------------------------------------- calls

def _create(A):
    """A device CSR to the library's tiled matrix."""
    h = ctypes.c_void_p()
    MF.check(MF.lib().mf_matrix_create(A.n, A.n, A.rowptr.data_ptr(), A.colidx.data_ptr(), A.val.data_ptr(), None, 1,
                                       None, ctypes.byref(h)))
    return MF.Matrix(None, _handle=h)


def _batch(A, sizes):
    rowptr, colidx, val = A.rowptr.cpu().numpy(), A.colidx.cpu().numpy(), A.val.cpu().numpy()
    systems, r = [], 0
    for n in sizes:
        lo, hi = rowptr[r], rowptr[r + n]
        systems.append(MF.HostCsr(n, n, rowptr[r:r + n + 1] - lo, colidx[lo:hi] - r, val[lo:hi]))
        r += n
    return MF.Batch(systems)


def prepare(case, seed):
    A = _matrix(case, seed)
    X = _columns(case, A.n, seed)
    call = case["call"]
    state = {"case": case, "n": A.n}
    if call in ("spmv", "spmm", "spmm_f16"):
        state.update(M=_create(A), x=X, y=torch.zeros_like(X))
    elif call == "build":
        state.update(A=A, x=X, y=torch.zeros_like(X))
    else:
        state.update(b=torch.stack([A.times(x) for x in X]), x=torch.zeros_like(X))
        opts = dict(tol=TOL[case["matrix"]], maxiter=MAXITER)
        if call == "batch":
            state["batch"] = _batch(A, _sizes(case))
            if case["policy"] == "learned":
                state["batch"].attach_policy(MF.Policy.load(PKG_DIR / "policies" / "randspd_batched.mfpol"))
            state["opts"] = dict(opts, policy=case["policy"])
        else:
            state["M"] = _create(A)
            state["opts"] = MF.solve_opts(policy=case.get("policy", "fp64"), **opts)
            state["report"] = (MF.SolveReport * case.get("k", 1))()
    return state


def run(state):
    L, case, n, call = MF.lib(), state["case"], state["n"], state["case"]["call"]
    stream = torch.cuda.current_stream().cuda_stream
    x, k = state["x"], case.get("k", 1)
    if call == "spmv":
        MF.check(L.mf_spmv(state["M"].h, x.data_ptr(), state["y"].data_ptr(), stream))
        return state["y"]
    if call == "spmm":
        MF.check(L.mf_spmm(state["M"].h, k, x.data_ptr(), n, state["y"].data_ptr(), n, stream))
        return state["y"]
    if call == "spmm_f16":
        MF.check(L.mf_spmm_f16(state["M"].h, k, x.data_ptr(), n, state["y"].data_ptr(), n, 0, None, stream))
        return state["y"]
    if call == "build":
        M = _create(state["A"])
        MF.check(L.mf_spmv(M.h, x.data_ptr(), state["y"].data_ptr(), stream))
        M.close()
        return state["y"]
    b = state["b"].data_ptr()
    if call == "batch":
        status, _ = state["batch"].solve_device(b, x.data_ptr(), use_graph=1, stream=stream, **state["opts"])
    elif call == "cg_multi":
        status = L.mf_cg_solve_multi(state["M"].h, k, b, n, x.data_ptr(), n, ctypes.byref(state["opts"]),
                                     state["report"], stream)
    else:
        solve = L.mf_bicgstab_solve if call == "bicgstab" else L.mf_cg_solve
        status = solve(state["M"].h, b, x.data_ptr(), ctypes.byref(state["opts"]), state["report"], None, stream)
    MF.check(status)
    return x


def exact(case, seed):
    A = _matrix(case, seed)
    X = _columns(case, A.n, seed)
    if case["call"] in ("spmv", "spmm", "spmm_f16", "build"):
        return torch.stack([A.times(x) for x in X])
    return X


# -------------------------------------------------------------------- work

def _shape(case):
    """(rows, entries) of a case's matrix, the random families' expected."""
    if case["call"] == "batch":
        lo, hi = case["n_min"], case["n_max"]
        n = case["systems"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        return n, 41 * n
    if case["matrix"] == "random_spd":
        return case["n"], 41 * case["n"]
    if case["matrix"] == "block_dense":
        return case["n"], 68 * case["n"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    cut = 2 * n * ((nx > 0) / nx + (ny > 0) / ny + ((1 / nz) if case["matrix"] != "lap2d" else 0))
    return n, (5 if case["matrix"] == "lap2d" else 7) * n - cut


def _iterations(case):
    """Iterations a solve of this size takes to the tolerances above
    (measured once with the FP64 solver, fitted)."""
    if case["matrix"] == "lap2d":
        return 3.7 * math.sqrt(case["nx"] * case["ny"])
    if case["matrix"] == "poisson3d":
        return 870.0
    if case["matrix"] == "convdiff3d":
        return 2.25 * max(case["nx"], case["ny"], case["nz"])
    return 17.0 * math.sqrt(case.get("n_max", case.get("n", 0)) * 0.5)


def work(case):
    n, nnz = _shape(case)
    k = case.get("k", 1)
    call = case["call"]
    if call in ("spmv", "spmm", "spmm_f16"):
        value = 2 if call == "spmm_f16" else 8
        return {"bytes": nnz * (value + 1) + 16 * n * k, "flops": 2 * nnz * k}
    if call == "build":
        return {"bytes": nnz * (12 + 9) + nnz * 9 + 20 * n, "flops": 2 * nnz}
    it = _iterations(case)
    low = case.get("policy", "fp64") != "fp64"
    value = 8 if not low else (2 if case["policy"] == "learned" else 4)
    index = 2 if call == "batch" else 1
    vectors = (36 if low else 72) * n * k
    products = 2 if call == "bicgstab" else 1
    return {"bytes": it * (products * nnz * (value + index) + vectors),
            "flops": it * k * (products * 2 * nnz + 10 * n)}


# ------------------------------------------------------------------- cases

def _case(name, call, matrix, **more):
    return dict(name=name, call=call, matrix=matrix, **more)


def listed():
    return [
        _case("spmv lap2d 128", "spmv", "lap2d", nx=128, ny=128, nz=1),
        _case("spmv poisson3d 128", "spmv", "poisson3d", nx=128, ny=128, nz=128),
        _case("spmm k5 convdiff odd", "spmm", "convdiff3d", nx=61, ny=67, nz=71, k=5),
        _case("spmm_f16 k16 blocks", "spmm_f16", "block_dense", n=262144, k=16),
        _case("build poisson3d 96", "build", "poisson3d", nx=96, ny=96, nz=96),
        _case("cg fp64 lap2d 128", "cg", "lap2d", nx=128, ny=128, nz=1, policy="fp64"),
        _case("cg fp64 poisson3d 128", "cg", "poisson3d", nx=128, ny=128, nz=128, policy="fp64"),
        _case("cg static poisson3d 128", "cg", "poisson3d", nx=128, ny=128, nz=128, policy="static"),
        _case("bicgstab static convdiff 96", "bicgstab", "convdiff3d", nx=96, ny=96, nz=96, policy="static"),
        _case("cg_multi k16 poisson3d 96", "cg_multi", "poisson3d", nx=96, ny=96, nz=96, k=16),
        _case("batch static small", "batch", "random_spd", systems=24, n_min=1000, n_max=4000, policy="static"),
        _case("batch learned", "batch", "random_spd", systems=256, n_min=1000, n_max=32000, policy="learned"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _grid(rng, lo, hi, flat):
    """Grid sides about the cube root (or square root) of a log-uniform size."""
    n = _log(rng, lo, hi)
    side = n ** (1 / 2 if flat else 1 / 3)
    nx = max(3, int(side * rng.uniform(0.7, 1.3)))
    ny = max(3, int(side * rng.uniform(0.7, 1.3)))
    nz = 1 if flat else max(3, n // (nx * ny))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    call = rng.choice(["spmv", "spmm", "spmm_f16", "build", "cg", "cg", "bicgstab", "cg_multi", "batch", "batch"])
    if call == "batch":
        lo = _log(rng, 500, 4000)
        return dict(call=call, matrix="random_spd", systems=_log(rng, 8, 160), n_min=lo,
                    n_max=_log(rng, lo + 1, 24000), policy=rng.choice(["static", "rule", "learned"]))
    if call == "spmm_f16":
        return dict(call=call, matrix="block_dense", n=_log(rng, 8000, 262144), k=rng.choice([1, 4, 7, 8, 13, 16]))
    case = dict(call=call, matrix=rng.choice(["lap2d", "poisson3d"]))
    if call in ("spmv", "spmm", "build"):
        case["matrix"] = rng.choice(["lap2d", "poisson3d", "convdiff3d", "random_spd"])
    if call == "bicgstab":
        case["matrix"] = "convdiff3d"
    if call in ("spmm", "cg_multi"):
        case["k"] = rng.choice([2, 3, 4, 5, 8, 11, 16])
    if call in ("cg", "bicgstab"):
        case["policy"] = rng.choice(["fp64", "static"])
    if call == "cg":
        case["matrix"] = rng.choice(["lap2d", "poisson3d", "poisson3d", "random_spd"])
    if case["matrix"] == "random_spd":
        return dict(case, n=_log(rng, 2000, 20000 if call == "cg" else 200000))
    top = {"cg_multi": 400000, "bicgstab": 880000, "build": 1000000}.get(call, 2000000)
    if case["matrix"] == "lap2d" and call in ("cg", "cg_multi"):
        top = 100000
    return dict(case, **_grid(rng, 4000, top, case["matrix"] == "lap2d"))
