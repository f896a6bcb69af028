"""mf_spmm_f16 where dense tiles and single entries alternate: rows with 0 to
40 single entries left of, between and right of a strip's dense tiles (the
kernel keeps 8 of a row's at a time), strips without either, a last strip of 1
to 15 rows, a last tile column of 1 to 15 columns.  Entries and X are small
integers, exact in FP16, and every partial sum is below 2^24: Y is exact."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def integer_matrix(rows, cols, seed):
    rng = np.random.default_rng(seed)
    A = np.zeros((rows, cols))
    for s in range(0, rows, 16):
        h = min(16, rows - s)
        for c in rng.choice(cols // 16, size=min(cols // 16, int(rng.integers(0, 5))), replace=False):  # dense tiles
            A[s:s + h, 16 * c:16 * c + 16] = rng.integers(1, 8, size=(h, 16))
        for r in range(s, s + h):
            n = min(cols, int(rng.choice([0, 0, 1, 3, 7, 8, 9, 16, 17, 40]))) if s % 48 != 32 else 0
            at = rng.choice(cols, size=n, replace=False)
            A[r, at] = rng.integers(1, 8, size=n)
    return A


@pytest.mark.parametrize("rows,cols", [(1, 17), (16, 2000), (95, 1311), (481, 1999)])
@pytest.mark.parametrize("k", [1, 8, 9, 16])
def test_alternating_tiles_exact(mf, rows, cols, k):
    import scipy.sparse as sp

    A = integer_matrix(rows, cols, rows + k)
    S = sp.csr_matrix(A)
    M = mf.Matrix(mf.HostCsr(rows, cols, S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data))
    X = np.random.default_rng(k).integers(-8, 9, size=(k, cols)).astype(np.float64)
    dX = torch.from_numpy(X).cuda()
    for fill in (1, 100, 256):  # all tiles dense, the full ones (of a short last strip: none), the full ones
        Y = torch.full((k, rows), np.nan, dtype=torch.float64, device="cuda")
        nd = C.c_int(-1)
        assert mf.lib().mf_spmm_f16(M.h, k, dX.data_ptr(), cols, Y.data_ptr(), rows, fill, C.byref(nd), None) == 0
        torch.cuda.synchronize()
        tiles = np.unique((S.tocoo().row // 16).astype(np.int64) * 4096 + S.tocoo().col // 16, return_counts=True)[1]
        assert nd.value == int(np.count_nonzero(tiles >= fill))
        assert np.array_equal(Y.cpu().numpy().T, A @ X.T)
    M.close()
