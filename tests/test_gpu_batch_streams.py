"""A batch's first solve on a stream that does not wait for the legacy default
stream (needs a B200): its workspace is zeroed in front of it, whatever the
default stream is busy with."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", ["fp64", "static"])
@pytest.mark.parametrize("cycles", [2_000_000, 10_000_000, 40_000_000])  # about 1, 5 and 20 ms
def test_first_solve_beside_a_busy_default_stream(mf, policy, cycles):
    A = [mf.synth_random_spd(50 + s, 30000) for s in range(4)]  # vectors in global memory
    b = torch.from_numpy(np.concatenate([M.matvec(mf.synth_xstar(s, M.n_rows)) for s, M in enumerate(A)])).cuda()
    B = mf.Batch(A)
    s = torch.cuda.Stream()
    xs = [torch.zeros_like(b) for _ in range(2)]
    torch.cuda.synchronize()
    torch.cuda._sleep(cycles)
    for x in xs:
        st, rep = B.solve_device(b.data_ptr(), x.data_ptr(), use_graph=0, stream=s.cuda_stream, tol=1e-10,
                                 maxiter=20000, policy=policy)
        assert st == 0 and rep.relres_true_max <= 1.2e-10
    torch.cuda.synchronize()
    assert torch.equal(xs[0], xs[1])
    B.close()
