"""mf_spmv from the row slots (a handle's later calls) against its first call,
which runs from the tiles (needs a B200): bit-identical on every edge-case
matrix, under stream capture, from two threads, and after a solve."""
import threading

import numpy as np
import pytest
import torch

import matrices

pytestmark = pytest.mark.gpu


def _wrapped(mf):
    """A tile of 256 entries (duplicates) whose last eight rows are empty --
    its last row pointers wrap to 0 -- beside rows of other lengths."""
    rng = np.random.default_rng(5)
    rows = [[(int(c), float(rng.normal())) for c in np.repeat(np.arange(16), 2)] for _ in range(8)]
    rows += [[] for _ in range(8)]
    for i in range(16, 40):
        rows.append([(int(c), float(rng.normal())) for c in rng.integers(0, 40, size=i % 11)])
    for i in range(0, 40, 3):
        rows[i] = rows[i] + [(35, float(rng.normal()))]
    rp = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    flat = [e for r in rows for e in r]
    return mf.HostCsr(40, 40, rp, np.array([c for c, _ in flat], np.int32), np.array([v for _, v in flat]))


def _all(mf):
    mats = {k: mf.HostCsr(A.n_rows, A.n_cols, A.rowptr, A.colidx, A.val) for k, A in matrices.all_matrices(mf).items()}
    mats["wrapped_tile"] = _wrapped(mf)
    mats["random_3001"] = mf.synth_random_spd(41, 3001)
    mats["convdiff_17"] = mf.synth_convdiff3d(17)
    return mats


def test_slots_equal_tiles_bit_for_bit(mf):
    L = mf.lib()
    for name, A in _all(mf).items():
        M = mf.Matrix(A)
        n = M.info().tilen * 16
        x = torch.from_numpy(np.sin(0.37 * np.arange(n) + 0.1) - 0.01 * np.arange(n)).cuda()
        ys = [torch.full((max(A.n_rows, 1),), 9.0, dtype=torch.float64, device="cuda") for _ in range(4)]
        for y in ys:
            mf.check(L.mf_spmv(M.h, x.data_ptr(), y.data_ptr(), None))
        torch.cuda.synchronize()
        for y in ys[1:]:
            assert torch.equal(y.view(torch.int64), ys[0].view(torch.int64)), name
        M.close()


def test_capture_and_threads(mf):
    L = mf.lib()
    A = mf.synth_poisson3d_scaled(20, 3)
    M = mf.Matrix(A)
    x = torch.from_numpy(mf.synth_xstar(4, A.n_rows)).cuda()
    y0, y1 = torch.zeros_like(x), torch.zeros_like(x)
    mf.check(L.mf_spmv(M.h, x.data_ptr(), y0.data_ptr(), None))
    torch.cuda.synchronize()
    # captured before the slots exist: served from the tiles, nothing allocated
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = torch.cuda.current_stream().cuda_stream
        for _ in range(3):
            mf.check(L.mf_spmv(M.h, x.data_ptr(), y1.data_ptr(), st))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y0, y1)
    outs = [torch.zeros_like(x) for _ in range(8)]
    streams = [torch.cuda.Stream() for _ in outs]

    def work(k):
        for _ in range(5):
            mf.check(L.mf_spmv(M.h, x.data_ptr(), outs[k].data_ptr(), streams[k].cuda_stream))

    th = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    [t.start() for t in th]
    [t.join() for t in th]
    torch.cuda.synchronize()
    assert all(torch.equal(o, y0) for o in outs)
    g.replay()
    xs, rep = M.solve_host(A.matvec(mf.synth_xstar(4, A.n_rows)), tol=1e-10, maxiter=3000)
    assert rep.status == 0
    mf.check(L.mf_spmv(M.h, x.data_ptr(), y1.data_ptr(), None))
    torch.cuda.synchronize()
    assert torch.equal(y0, y1)
    M.close()
