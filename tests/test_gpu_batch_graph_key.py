"""A batch's kept CUDA graph (needs a B200): a solve with other options on the
same buffers is not a replay of the last one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tols", [(1e-3, 1e-5), (1e-5, 1e-3), (1e-13, 0.9e-13), (4e-16, 1e-6)])
def test_tolerance_is_part_of_the_key(mf, tols):
    A = [mf.synth_random_spd(100 + s, 1200 + 100 * s) for s in range(3)]
    b = torch.from_numpy(np.concatenate([M.matvec(mf.synth_xstar(s, M.n_rows)) for s, M in enumerate(A)])).cuda()
    x = torch.zeros_like(b)
    B, F = mf.Batch(A), mf.Batch(A)
    for tol in tols:
        # a tolerance that FP64 cannot reach ends at maxiter: the same with and without a graph
        st, rep = B.solve_device(b.data_ptr(), x.data_ptr(), use_graph=1, tol=tol, maxiter=300, policy="fp64")
        y = x.clone()
        sf, want = F.solve_device(b.data_ptr(), x.data_ptr(), use_graph=0, tol=tol, maxiter=300, policy="fp64")
        assert st == sf and rep.iterations_total == want.iterations_total
        assert torch.equal(x, y)
        if st == 0:
            assert rep.relres_true_max <= 1.2 * tol
    B.close()
    F.close()


def test_refine_delta_is_part_of_the_key(mf):
    A = [mf.synth_random_spd(7, 1500)]
    b = torch.from_numpy(A[0].matvec(mf.synth_xstar(3, 1500))).cuda()
    x = torch.zeros_like(b)
    B = mf.Batch(A)
    refs = []
    for delta in (1e-3, 1e-3 + 4e-7, 1e-1):
        st, rep = B.solve_device(b.data_ptr(), x.data_ptr(), use_graph=1, tol=1e-10, maxiter=2000, policy="static",
                                 refine_delta=delta)
        sf, want = B.solve_device(b.data_ptr(), x.data_ptr(), use_graph=0, tol=1e-10, maxiter=2000, policy="static",
                                  refine_delta=delta)
        assert st == sf == 0 and rep.refinements_total == want.refinements_total
        refs.append(rep.refinements_total)
    assert refs[-1] > refs[0]
    B.close()
