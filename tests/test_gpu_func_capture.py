"""exp and its adjoint of one matrix inside a stream that the caller captures, at sizes below and
from the one where the whole GPU takes over (96): replays see what the buffers hold then."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
sl = pytest.importorskip("scipy.linalg")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _skew(n, seed):
    B = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    return B - B.T


@pytest.mark.parametrize("n", [40, 96, 200, 700])
def test_replay(skewgpu, n):
    L = skewgpu._lib.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    W, E, C, G = (torch.zeros_like(A) for _ in range(4))
    info = torch.zeros(1, dtype=torch.int32, device="cuda")

    def both(h):
        W.copy_(A)
        assert L.skew_exp_d(h, p(W), n, n, p(E), n, p(info)) == 0
        W.copy_(A)
        assert L.skew_exp_vjp_d(h, p(W), n, n, p(C), p(G), n, p(info)) == 0

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        h = skewgpu.handle().bind()
        both(h)  # workspaces at their size
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
            both(h)
    for seed in (1, 2):
        M, D = _skew(n, seed), np.random.default_rng(10 + seed).standard_normal((n, n))
        A.copy_(skewgpu.to_device(M))
        C.copy_(skewgpu.to_device(D))
        E.zero_()
        G.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert int(info.item()) == 0
        want = sl.expm(M)
        assert np.linalg.norm(E.cpu().numpy().T - want) <= 40 * n * EPS * np.linalg.norm(want)
        if n <= 200:
            want = sl.expm_frechet(M.T, D, compute_expm=False)
            assert np.linalg.norm(G.cpu().numpy().T - want) <= 40 * n * EPS * np.linalg.norm(want)
