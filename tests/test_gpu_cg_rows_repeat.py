"""FP64 CG with the rows in registers (needs a B200): every solve of a system
gives the same bits, in as many iterations (all CTAs must see the same partial
sums at every grid-wide reduction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [130, 200, 275])  # 67 to 296 CTAs
def test_repeated_solves_are_identical(mf, side):
    A = mf.synth_laplace2d(side, side)
    b = A.matvec(mf.synth_xstar(1, A.n_rows))
    M = mf.Matrix(A)
    x0, r0 = M.solve_host(b, tol=1e-12, maxiter=5000)
    assert r0.status == 0
    for _ in range(20):
        x, r = M.solve_host(b, tol=1e-12, maxiter=5000)
        assert r.iterations == r0.iterations and np.array_equal(x, x0)
    M.close()
