"""The mixed batched solver's sorted slices where they can go wrong (needs a
B200): rows spread over a warp (256 entries and more), rows without
off-diagonal entries, a last slice of one row, systems on both sides of the
on-chip limit and of one column window, every cluster size, every policy,
against the FP64 CPU oracle."""
import numpy as np
import pytest
import torch

import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _arrow(mf, n, dense, seed):
    """SPD: `dense` full rows and columns, a chain, and isolated rows."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    B = sp.lil_matrix((n, n))
    for d in range(dense):
        cols = rng.choice(n, size=min(n, 255 + 3 * d + (d % 2)), replace=False)
        B[d, cols] = rng.normal(size=cols.size)
    for i in range(n // 2, n - 7):
        B[i, i + 1] = rng.normal()
    B = B.tocsr()
    A = (B + B.T) * 0.5
    A.setdiag(0)
    A.eliminate_zeros()
    A = A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)
    A = A.tocsr()
    A.sort_indices()
    return mf.HostCsr(n, n, A.indptr, A.indices, A.data)


@pytest.fixture(scope="module")
def problems(mf):
    systems = [_arrow(mf, 1025, 9, 1), _arrow(mf, 300, 40, 2), mf.synth_random_spd(11, 33), mf.synth_random_spd(12, 2049),
               mf.synth_random_spd(13, 22200), mf.synth_random_spd(14, 55400), mf.synth_laplace2d(37, 29)]
    xs = [mf.synth_xstar(20 + k, A.n_rows) for k, A in enumerate(systems)]
    bs = [A.matvec(x) for A, x in zip(systems, xs)]
    oracle = []
    for A, b, x in zip(systems, bs, xs):
        Ac = ol.Csr(A.n_rows, A.n_cols, A.rowptr, A.colidx, A.val)
        it, x_o, _ = ol.oracle_cg(Ac, b, 50000, 1e-10)
        oracle.append((Ac, it, x_o, np.max(np.abs(x_o - x))))
    return systems, bs, oracle


@pytest.mark.parametrize("cluster,policy", [(1, "static"), (2, "rule"), (2, "learned"), (4, "static"), (8, "learned"),
                                            (16, "rule")])
def test_slices_match_oracle(mf, problems, cluster, policy):
    from pathlib import Path

    systems, bs, oracle = problems
    B = mf.Batch(systems)
    mf.check(mf.lib().mf_batch_set_schedule(B.h, 4, cluster))
    P = mf.Policy.load(Path(__file__).resolve().parent.parent / "mille-feuille_b200" / "policies" /
                       "randspd_batched.mfpol")
    B.attach_policy(P if policy == "learned" else None)
    db = torch.from_numpy(B.stack(bs)).cuda()
    dx = torch.full_like(db, 3.0)
    st, rep = B.solve_device(db.data_ptr(), dx.data_ptr(), use_graph=0, tol=1e-10, maxiter=50000, policy=policy)
    assert st == 0 and rep.failed == 0, rep.as_dict()
    first = dx.clone()
    its, _ = B.results()
    for k, (xk, (Ac, it_o, x_o, err_o)) in enumerate(zip(B.split(first.cpu().numpy()), oracle)):
        assert ol.oracle_true_relres(Ac, bs[k], xk) <= 1.2e-10, k
        assert np.max(np.abs(xk - x_o)) <= 100 * err_o + 1e-9, k
        assert its[k] <= 1.5 * it_o + 10, (k, its[k], it_o)
    st, rep2 = B.solve_device(db.data_ptr(), dx.data_ptr(), use_graph=0, tol=1e-10, maxiter=50000, policy=policy)
    assert st == 0 and torch.equal(first, dx) and rep2.bytes_moved == rep.bytes_moved
    B.close()
    P.close()
