"""A batch made, solved and destroyed on one thread while another thread captures
a stream (needs a B200): the graph is complete, the solve is right."""
import threading

import numpy as np
import torch

import pytest

pytestmark = pytest.mark.gpu


def test_batch_beside_another_threads_capture(mf):
    A = [mf.synth_random_spd(60 + s, 1500) for s in range(3)]
    b = torch.from_numpy(np.concatenate([M.matvec(mf.synth_xstar(s, 1500)) for s, M in enumerate(A)])).cuda()
    xs = [torch.zeros_like(b) for _ in range(2)]
    pol = mf.Policy(seed=3)
    s = torch.cuda.Stream()
    out = []

    def work(x):
        B = mf.Batch(A)
        B.attach_policy(pol)
        for policy in ("static", "learned", "fp64"):
            out.append(B.solve_device(b.data_ptr(), x.data_ptr(), use_graph=1, stream=s.cuda_stream, tol=1e-10,
                                      maxiter=5000, policy=policy)[0])
        B.close()

    work(xs[0])  # kernels loaded
    g, c = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    v = torch.ones(1000, device="cuda")
    y = torch.zeros_like(v)
    torch.cuda.synchronize()
    with torch.cuda.stream(c):
        g.capture_begin(capture_error_mode="thread_local")
        y.add_(v)
        t = threading.Thread(target=work, args=(xs[1],))
        t.start()
        t.join()
        y.add_(v)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert torch.all(y == 2.0)
    assert out == [0] * 6 and torch.equal(xs[0], xs[1])
