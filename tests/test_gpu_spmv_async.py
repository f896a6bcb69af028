"""mf_spmv never makes the host wait (needs a B200): not for the row slots
either, which a handle's second product queues on its stream.  Other streams,
captures and solves that come before they are complete give the same bits."""
import ctypes as C

import numpy as np
import pytest
import torch

import matrices

pytestmark = pytest.mark.gpu

SLEEP = 400_000_000  # clock cycles: about 0.2 s


def _long_rows(mf):
    """Rows of up to 400 entries (tile-rows above 256 entries), 32-bit distances."""
    rng = np.random.default_rng(6)
    n = 40000
    rows = [sorted(rng.choice(n, size=int(k), replace=False).tolist()) for k in rng.integers(0, 400, size=100)]
    rows += [[i] for i in range(100, n)]
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    ci = np.concatenate([np.array(r, np.int32) for r in rows])
    return mf.HostCsr(n, n, rp, ci, rng.normal(size=ci.size))


def _wrapped(mf):
    """A tile of 256 entries with an empty last row: its sizes are not known
    before the slots are counted."""
    rng = np.random.default_rng(5)
    rows = [np.repeat(np.arange(16), 2) for _ in range(8)] + [np.zeros(0, int) for _ in range(8)]
    rows += [np.array([3, 30]) for _ in range(24)]
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    return mf.HostCsr(40, 40, rp, np.concatenate(rows).astype(np.int32), rng.normal(size=rp[-1]))


def _mats(mf):
    return {"poisson": mf.synth_poisson3d_scaled(24, 3), "random": mf.synth_random_spd(9, 3001),
            "long_rows": _long_rows(mf), "wrapped": _wrapped(mf)}


def _setup(mf, name):
    A = _mats(mf)[name]
    M, T = mf.Matrix(A), mf.Matrix(A)
    x = torch.from_numpy(np.sin(0.37 * np.arange(M.info().tilen * 16) + 0.1)).cuda()
    want = torch.zeros(A.n_rows, dtype=torch.float64, device="cuda")
    mf.check(mf.lib().mf_spmv(T.h, x.data_ptr(), want.data_ptr(), None))  # a handle's first: from the tiles
    torch.cuda.synchronize()
    return A, M, T, x, want


@pytest.mark.parametrize("name", ["poisson", "random", "long_rows", "wrapped"])
def test_host_never_waits(mf, name):
    A, M, T, x, want = _setup(mf, name)
    for _ in range(2):  # once before the measured handle: kernels loaded
        L = mf.lib()
        a, b = torch.cuda.Stream(), torch.cuda.Stream()
        ys = [torch.full_like(want, 9.0) for _ in range(6)]
        done = torch.cuda.Event()
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(SLEEP)
            done.record()
        for y in ys[:4]:
            mf.check(L.mf_spmv(M.h, x.data_ptr(), y.data_ptr(), a.cuda_stream))
        for y in ys[4:]:
            mf.check(L.mf_spmv(M.h, x.data_ptr(), y.data_ptr(), b.cuda_stream))
        late = not done.query()
        torch.cuda.synchronize()
        for y in ys:
            assert torch.equal(y.view(torch.int64), want.view(torch.int64))
        M, T = T, M
    assert late
    M.close()
    T.close()


@pytest.mark.parametrize("name", ["poisson", "random"])
def test_capture_and_solve_before_the_slots_are_complete(mf, name):
    A, M, T, x, want = _setup(mf, name)
    L = mf.lib()
    a = torch.cuda.Stream()
    ys = [torch.full_like(want, 9.0) for _ in range(4)]
    Y = torch.zeros(2, A.n_rows, dtype=torch.float64, device="cuda")
    X = torch.stack([x[:A.n_rows], 2 * x[:A.n_rows]])
    mf.check(L.mf_spmm(T.h, 2, X.data_ptr(), A.n_rows, Y.data_ptr(), A.n_rows, None))  # kernels loaded
    b = torch.from_numpy(A.matvec(mf.synth_xstar(4, A.n_rows))).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(SLEEP)
    for y in ys[:2]:
        mf.check(L.mf_spmv(M.h, x.data_ptr(), y.data_ptr(), a.cuda_stream))
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        mf.check(L.mf_spmv(M.h, x.data_ptr(), ys[2].data_ptr(), s.cuda_stream))
        mf.check(L.mf_spmm(M.h, 2, X.data_ptr(), A.n_rows, Y.data_ptr(), A.n_rows, s.cuda_stream))
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y in ys[:3])
    assert torch.equal(Y[0], want) and torch.equal(Y[1], 2 * want)
    # a solve on another stream right behind the product that queues the slots
    N = mf.Matrix(A)
    xs = [torch.zeros_like(b) for _ in range(2)]
    rep = mf.SolveReport()
    opts = mf.solve_opts(tol=1e-10, maxiter=20000)
    mf.check(L.mf_cg_solve(T.h, b.data_ptr(), xs[0].data_ptr(), C.byref(opts), C.byref(rep), None, None))
    for y in ys[:2]:
        mf.check(L.mf_spmv(N.h, x.data_ptr(), y.data_ptr(), a.cuda_stream))
    mf.check(L.mf_cg_solve(N.h, b.data_ptr(), xs[1].data_ptr(), C.byref(opts), C.byref(rep), None, s.cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(xs[0], xs[1])
    for m in (M, T, N):
        m.close()


def test_device_bytes_count_the_slots(mf):
    A = mf.synth_poisson3d_scaled(24, 3)
    M = mf.Matrix(A)
    before = M.info().device_bytes
    x = torch.zeros(A.n_rows, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    for _ in range(2):
        mf.check(mf.lib().mf_spmv(M.h, x.data_ptr(), y.data_ptr(), None))
    torch.cuda.synchronize()
    assert M.info().device_bytes >= before + 12 * A.nnz
    M.close()


def test_slots_are_not_built_under_a_capture(mf):
    """mf_spmm's first call needs the slots: refused while its stream is captured
    (their memory would belong to the graph), and nothing of it stays."""
    A = mf.synth_poisson3d_scaled(12, 3)
    n = A.n_rows
    M, T = mf.Matrix(A), mf.Matrix(A)
    L = mf.lib()
    X = torch.from_numpy(np.random.default_rng(3).normal(size=(2, n))).cuda()
    Y, want = torch.zeros_like(X), torch.zeros_like(X)
    mf.check(L.mf_spmm(T.h, 2, X.data_ptr(), n, want.data_ptr(), n, None))
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        st = L.mf_spmm(M.h, 2, X.data_ptr(), n, Y.data_ptr(), n, s.cuda_stream)
        Y.add_(1.0)
        g.capture_end()
    assert st == 2  # MF_ERR_CUDA
    g.replay()
    torch.cuda.synchronize()
    assert torch.all(Y == 1.0)
    mf.check(L.mf_spmm(M.h, 2, X.data_ptr(), n, Y.data_ptr(), n, None))
    torch.cuda.synchronize()
    assert torch.equal(Y, want)
    M.close()
    T.close()


@pytest.mark.parametrize("tiles", [4096, 4097])
def test_strip_of_many_tiles(mf, tiles):
    """A strip of 4,096 tiles has slots, one more has none (a slot's word cannot
    name the tile): products from the tiles, mf_spmm refused."""
    n = 16 * tiles
    ci = 16 * np.arange(tiles) + np.arange(tiles) % 16
    rp = np.zeros(n + 1, np.int32)
    rp[6:] = tiles
    A = mf.HostCsr(n, n, rp, ci, np.random.default_rng(2).normal(size=tiles))
    M = mf.Matrix(A)
    L = mf.lib()
    x = torch.from_numpy(np.cos(0.1 * np.arange(n))).cuda()
    ys = [torch.full((n,), 9.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    for y in ys:
        mf.check(L.mf_spmv(M.h, x.data_ptr(), y.data_ptr(), None))
    X = torch.stack([x, x])
    Y = torch.zeros_like(X)
    st = L.mf_spmm(M.h, 2, X.data_ptr(), n, Y.data_ptr(), n, None)
    torch.cuda.synchronize()
    assert all(torch.equal(y, ys[0]) for y in ys[1:])
    assert abs(ys[0][5].item() - float(A.val @ np.cos(0.1 * ci))) <= 1e-10 * tiles
    assert st == (0 if tiles <= 4096 else 8)  # MF_ERR_UNSUPPORTED
    if st == 0:
        assert torch.equal(Y[0], ys[0]) and torch.equal(Y[1], ys[0])
    M.close()


def test_matrix_without_rows(mf):
    """No tile-row: every array with an end entry ends at 0."""
    M = mf.Matrix(mf.HostCsr(0, 40, [0], [], []))
    i = M.info()
    assert (i.rows, i.nnz, i.tilem, i.tilenum, i.csrptrlen, i.nonzero_rows) == (0, 0, 0, 0, 0, 0)
    for name in ("tile_nnz", "csrptr_offset", "blknnznnz", "nonzero_row_new"):
        assert not np.any(M.export(name))
    M.close()
