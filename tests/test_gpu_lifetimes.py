"""Memory of handles and calls: who may still be using it when it goes back."""
import numpy as np
import pytest

import chronoslab_b200 as cb
from chronoslab_b200 import problems as PB

pytestmark = pytest.mark.gpu


def _captured_cycle(h, b, x):
    import torch
    h.vcycle_dev(b.data_ptr(), x.data_ptr())
    torch.cuda.synchronize()
    want = x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        h.vcycle_dev(b.data_ptr(), x.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    x.zero_()
    return g, want


@pytest.mark.parametrize("beside_capture", [False, True])
def test_free_waits_for_replays(lib, beside_capture):
    """A handle freed with replays of its captured V-cycle still queued on the
    caller's stream, also while another capture is being taken: the free returns
    after the replays, and a handle set up in the memory it gave back does not
    reach their result."""
    import torch
    A = PB.poisson7(40)
    n = A.shape[0]
    prm = cb.params(precision=cb.CHRONOS_FP64, ntv=1)
    b = torch.from_numpy(np.random.default_rng(3).standard_normal(n)).cuda()
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    other = cb.Hierarchy(A, np.ones((n, 1)), prm)
    other.vcycle_dev(b.data_ptr(), y.data_ptr())
    h = cb.Hierarchy(A, np.ones((n, 1)), prm)
    g, want = _captured_cycle(h, b, x)
    run = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(run):
        for _ in range(400):
            g.replay()
    if beside_capture:
        g2 = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g2, capture_error_mode="relaxed"):
            other.vcycle_dev(b.data_ptr(), y.data_ptr(),
                             stream=torch.cuda.current_stream().cuda_stream)
            h.close()
    else:
        h.close()
    assert run.query()
    with cb.Hierarchy(2.0 * A, np.ones((n, 1)), prm) as h2:
        h2.pcg(b.cpu().numpy(), tol=1e-8)
    torch.cuda.synchronize()
    assert torch.equal(x, want)
    if beside_capture:
        y.zero_()
        g2.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    other.close()
