"""A plan's first batched gradient inside a stream that the caller captures: nothing is allocated
there, and the replayed graph gives the gradients of what the buffers hold."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("sizes", [[130, 16, 200], [98]])
def test_first_gradient_in_a_capture(skewgpu, sizes):
    mats = []
    for n in sizes:
        B = np.random.default_rng(n).standard_normal((n, n)) / np.sqrt(n)
        A = (B - B.T) / 2
        k = np.arange(0, n, 2)
        A[k, k + 1] += 2.0
        A[k + 1, k] -= 2.0
        mats.append(A)
    plan = skewgpu.BatchPlan(sizes)
    dA = [skewgpu.to_device(A) for A in mats]
    dG = [torch.zeros_like(a) for a in dA]
    pa, pg = plan.pointer_array(dA), plan.pointer_array(dG)
    out = [torch.zeros(len(sizes), dtype=torch.float64, device="cuda") for _ in range(2)]
    st = torch.zeros(len(sizes), dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        plan.logabspfaffian(pa, None, *out, st)  # without gradients: binds the handle to s
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
            plan.logabspfaffian(pa, pg, *out, st)
    for _ in range(2):
        for G in dG:
            G.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        for A, G in zip(mats, dG):
            want = np.linalg.inv(A).T / 2
            # well-conditioned: a modest multiple of n eps
            assert np.linalg.norm(skewgpu.from_device(G) - want) <= 20 * len(A) * EPS * np.linalg.norm(want)
        plan.logabspfaffian(pa, pg, *out, st)  # outside: takes its workspace, the graph stays good
    plan.close()
