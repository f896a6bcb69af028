"""The tile build around its size limits (needs a B200): tile-rows of 0 to 300
entries -- one warp's 32, 64, 128 and 256 keys and the block path above --
with unsorted and duplicate columns, a ragged last tile-row, and values of
every class, against the CPU oracle's tiles and NumPy's payloads, bit for
bit."""
import numpy as np
import pytest

import oracle_lib as ol

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 255, 256, 257, 300]


def _matrix(rows_last, cols, seed, order):
    rng = np.random.default_rng(seed)
    per_row = []
    for m in [SIZES[k] for k in order]:
        cut = np.sort(rng.integers(0, m + 1, 15))
        per_row += np.diff(np.concatenate([[0], cut, [m]])).tolist()
    per_row += rng.integers(0, 9, rows_last).tolist()
    rp = np.concatenate([[0], np.cumsum(per_row)]).astype(np.int32)
    nnz = int(rp[-1])
    ci = rng.integers(0, cols, nnz).astype(np.int32)  # unsorted, some repeated
    kind = rng.integers(0, 5, nnz)
    v = np.where(kind == 0, rng.integers(-128, 128, nnz).astype(np.float64), rng.normal(size=nnz))
    v = np.where(kind == 1, np.float16(rng.normal(size=nnz)).astype(np.float64), v)
    v = np.where(kind == 2, np.float32(rng.normal(size=nnz)).astype(np.float64), v)
    v = np.where(kind == 3, rng.normal(size=nnz) * 10.0 ** rng.uniform(-12, 12, nnz), v)
    # whole tile-rows of one kind too, so that every class occurs
    for k, m in enumerate(order):
        a, b = rp[16 * k], rp[16 * k + 16]
        if k % 4 == 0:
            v[a:b] = rng.integers(-128, 128, b - a)
        elif k % 4 == 1:
            v[a:b] = np.float16(rng.normal(size=b - a))
        elif k % 4 == 2:
            v[a:b] = np.float32(rng.normal(size=b - a))
    return ol.Csr(len(per_row), cols, rp, ci, v)


@pytest.mark.parametrize("rows_last,cols,seed", [(0, 900, 1), (5, 70, 2), (15, 4000, 3), (1, 257, 4)])
def test_tile_build_sizes(mf, rows_last, cols, seed):
    order = np.random.default_rng(seed + 100).permutation(len(SIZES))
    A = _matrix(rows_last, cols, seed, order)
    M = mf.Matrix(mf.HostCsr(A.n_rows, A.n_cols, A.rowptr, A.colidx, A.val))
    sizes, arrs, t = ol.oracle_tiles(A)
    try:
        inf = M.info()
        assert inf.tilenum == sizes["tilenum"] and inf.csrptrlen == sizes["csrptrlen"]
        for k, want in arrs.items():
            assert np.array_equal(M.export(k), want), k
        tn = M.export("tile_nnz").astype(np.int64)
        val, low = M.export("Blockcsr_Val"), M.export("Blockcsr_Val_Low")
        with np.errstate(over="ignore", invalid="ignore"):
            h = low.astype(np.float16)
            f32 = val.astype(np.float32).astype(np.float64)
        assert np.array_equal(M.export("payload_f16"), h.view(np.uint16))
        whole = (val == np.trunc(val)) & (val >= -128) & (val <= 127)
        assert np.array_equal(M.export("payload_i8")[whole], val[whole].astype(np.int8))
        cls, ok = M.export("tile_class"), M.export("tile_f16ok")
        for k in range(inf.tilenum):
            e = slice(tn[k], tn[k + 1])
            want = 2 if whole[e].all() else 3 if (h[e].astype(np.float64) == val[e]).all() else (
                4 if (f32[e] == val[e]).all() else 0)
            assert cls[k] == want, k
            fin = np.isfinite(h[e]).all()
            norm = (np.abs(h[e][val[e] != 0].astype(np.float64)) >= 2.0 ** -14).all()
            assert ok[k] == (1 if fin else 0) + (2 if fin and norm else 0), k
        assert list(inf.class_tiles) == [int((cls == c).sum()) for c in range(5)]
        assert inf.max_tile_nnz == int(np.diff(tn).max())
    finally:
        ol.free_oracle_tiles(t)
        M.close()
