"""FP64 CG with the rows in registers (needs a B200) at the edges of its
range: one row to 75,776 (the most resident threads) and one more, rows of 8
entries and of 9 (the chunked kernel), distances beyond 16 bits, a fixed
iteration count, a zero right-hand side; against the FP64 CPU oracle."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _banded(mf, n, offsets, seed):
    """SPD: random couplings at the given distances, diagonal |sum| + 1."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    A = sp.csr_matrix((n, n))
    for o in offsets:
        if o < n:
            v = rng.normal(size=n - o)
            A = A + sp.diags([v, v], [-o, o], shape=(n, n))
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsr()
    A.sort_indices()
    return mf.HostCsr(n, n, A.indptr, A.indices, A.data)


@pytest.mark.parametrize("n,offsets", [
    (1, [1]), (15, [1]), (16, [1, 3]), (17, [2]), (255, [1, 16, 17]), (256, [1, 15]), (257, [1, 5, 90]),
    (5000, [1, 7, 400]),            # 7 entries per row
    (5000, [1, 7, 400, 4900]),      # 9 at most: the chunked kernel
    (75000, [1, 40000]),            # 32-bit distances
    (75776, [1, 270]), (75777, [1, 270]),
])
def test_rows_cg_matches_oracle(mf, n, offsets):
    A = _banded(mf, n, offsets, n + len(offsets))
    xs = mf.synth_xstar(n, n)
    b = A.matvec(xs)
    Ac = ol.Csr(n, n, A.rowptr, A.colidx, A.val)
    it_o, x_o, _ = ol.oracle_cg(Ac, b, 5000, 1e-10)
    M = mf.Matrix(A)
    x, rep = M.solve_host(b, tol=1e-10, maxiter=5000)
    assert rep.status == 0
    assert abs(rep.iterations - it_o) <= max(3, it_o // 50)
    assert ol.oracle_true_relres(Ac, b, x) <= 1.2e-10
    assert np.max(np.abs(x - x_o)) <= 100 * np.max(np.abs(x_o - xs)) + 1e-12
    x2, _ = M.solve_host(b, tol=1e-10, maxiter=5000)
    assert np.array_equal(x, x2)
    # a fixed count of iterations, and a zero right-hand side
    k = min(5, max(1, it_o - 1))
    x3, rep3 = M.solve_host(b, tol=-1.0, maxiter=k)
    _, x_k, _ = ol.oracle_cg(Ac, b, k, -1.0)
    if n > 1:
        assert rep3.iterations == k
    assert np.max(np.abs(x3 - x_k)) <= 1e-11 * max(1.0, np.max(np.abs(x_k)))
    x4, rep4 = M.solve_host(np.zeros(n), tol=1e-10, maxiter=10)
    assert rep4.iterations == 0 and np.all(x4 == 0.0)
    M.close()
