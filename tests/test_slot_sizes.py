"""The row slots' sizes as the build of the tiles takes them from the CSR rows
(the longest row of every strip, the farthest tile) against the tiles' own row
bounds, from which the slots are filled: alike unless a tile of 256 entries has
an empty last row (its 8-bit row pointers wrap, and rows get other entries)."""
import numpy as np

import matrices
import oracle_lib as ol


def wrapped():
    rng = np.random.default_rng(5)
    rows = [[(int(c), float(rng.normal())) for c in np.repeat(np.arange(16), 2)] for _ in range(8)]
    rows += [[] for _ in range(8)] + [[(3, 1.0)]] * 5
    return matrices._from_rows(21, 40, rows)


def full_last_row():
    """A tile of 256 entries, all in its last row: nothing wraps."""
    return matrices._from_rows(16, 20, [[] for _ in range(15)] + [[(c, 1.0) for c in range(16)] * 16])


def long_rows():
    rng = np.random.default_rng(6)
    rows = [sorted(rng.choice(3000, size=int(k), replace=False).tolist()) for k in rng.integers(0, 400, size=70)]
    return matrices._from_rows(70, 3000, [[(c, 1.0) for c in r] for r in rows])


def _check(name, A):
    sizes, t, keep = ol.oracle_tiles(A)
    length = np.diff(A.rowptr)
    total = total_t = kmax_t = far = far_t = 0
    odd = False
    for s in range(sizes["tilem"]):
        lo, hi = 16 * s, min(A.n_rows, 16 * s + 16)
        total += int(length[lo:hi].max())
        cols = A.colidx[A.rowptr[lo]:A.rowptr[hi]] // 16
        far = max([far] + np.abs(s - cols).tolist())
        rows = np.zeros(hi - lo, np.int64)
        for k in range(t["tile_ptr"][s], t["tile_ptr"][s + 1]):
            nz = int(t["tile_nnz"][k + 1] - t["tile_nnz"][k])
            p = t["Blockcsr_Ptr"][t["csrptr_offset"][k]:][:hi - lo].astype(int).tolist() + [nz]
            rows += np.maximum(np.diff(p), 0)
            odd |= nz == 256 and not np.any((A.colidx[A.rowptr[hi - 1]:A.rowptr[hi]] // 16) == t["tile_columnidx"][k])
            far_t = max(far_t, abs(s - int(t["tile_columnidx"][k])))
        total_t += int(rows.max())
        kmax_t = max(kmax_t, int(rows.max()))
    ol.free_oracle_tiles(keep)
    assert odd == (name == "wrapped")
    if not odd:
        assert (total, int(length.max(initial=0)), far) == (total_t, kmax_t, far_t)


def test_sizes_from_rows_equal_sizes_from_tiles(mf):
    cases = dict(matrices.all_matrices(mf), wrapped=wrapped(), full_last_row=full_last_row(), long_rows=long_rows())
    for name, A in cases.items():
        _check(name, A)
