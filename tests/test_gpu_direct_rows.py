"""FP64 CG (plain and Jacobi) and BiCGSTAB with a thread per row straight from
the slot arrays (needs a B200), against the same solve from the staged slot
chunks: rows of 3 to 65 entries (batches of 8, or 6 for three vectors, and
every remainder), the longest on both sides of 4 times the average, distances
beyond 16 bits, short last strips, empty off-diagonals.  Six iterations of a
diagonally dominant system: the rows' sums are the same bits, the dot products
differ in order, a few 1e-16 per iteration."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(mf, n, half, longest, span, seed):
    """Symmetric, up to `half` entries per row and side within `span`; one row
    and column of `longest` entries; dominant diagonal."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    lens = rng.integers(0, half + 1, n)
    rows = np.repeat(np.arange(n), lens)
    cols = np.minimum(rows + 1 + rng.integers(0, span, rows.size), n - 1)
    at = rng.choice(n, size=longest, replace=False)
    rows, cols = np.r_[rows, np.full(longest, n // 2)], np.r_[cols, at]
    A = sp.csr_matrix((rng.normal(size=rows.size), (rows, cols)), shape=(n, n))
    A = A + A.T
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsr()
    A.sort_indices()
    return mf.HostCsr(n, n, A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)


@pytest.mark.parametrize("n,half,longest,span", [
    (16385, 3, 1, 40), (33001, 6, 1, 700),     # one reduction, up to 16 entries
    (1000, 9, 20, 100), (4097, 12, 60, 4000), (4097, 3, 62, 300),
    (20000, 16, 1, 90), (70000, 24, 1, 50000),  # 32-bit distances
    (66000, 40, 1, 500),                        # longest above 64
])
def test_direct_rows_match_chunks(mf, monkeypatch, n, half, longest, span):
    A = _matrix(mf, n, half, longest, span, n + half)
    b = np.random.default_rng(n).normal(size=n)
    M = mf.Matrix(A)
    for method, opts in (("cg", {}), ("cg", {"precond": 1}), ("bicgstab", {})):
        xs = []
        for layout in (None, "chunks"):
            if layout:
                monkeypatch.setenv("MF_SOLVER_LAYOUT", layout)
            else:
                monkeypatch.delenv("MF_SOLVER_LAYOUT", raising=False)
            x, rep = M.solve_host(b, method=method, tol=-1.0, maxiter=6, **opts)
            assert rep.iterations == 6
            xs.append(x)
        scale = np.max(np.abs(xs[1]))
        assert np.max(np.abs(xs[0] - xs[1])) <= 1e-13 * scale
        monkeypatch.delenv("MF_SOLVER_LAYOUT", raising=False)
        x2, _ = M.solve_host(b, method=method, tol=-1.0, maxiter=6, **opts)
        assert np.array_equal(xs[0], x2)
    M.close()
