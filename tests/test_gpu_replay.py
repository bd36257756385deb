"""Batched eigenvectors from the logged rotations: sizes at the edges of a warp's rows, odd and
even, in one batch and alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("sizes", [[1, 2, 3, 4, 5], [65, 64, 63, 62, 66], [130, 127, 1, 129, 128], [257]])
def test_eigenpairs(skewgpu, sizes):
    mats = []
    for n in sizes:
        B = np.random.default_rng(n).standard_normal((n, n))
        mats.append(B - B.T)
    dA = [skewgpu.to_device(A) for A in mats]
    plan = skewgpu.BatchPlan(sizes)
    f = lambda *s: torch.full(s, 7.0, dtype=torch.float64, device="cuda")
    v = [f(n) for n in sizes]
    re, im = [f(n, n) for n in sizes], [f(n, n) for n in sizes]
    st = plan.eigen(plan.pointer_array(dA), plan.pointer_array(v), plan.pointer_array(re), plan.pointer_array(im))
    assert (st.cpu().numpy() == 0).all()
    for n, A, w, x, y in zip(sizes, mats, v, re, im):
        lam = 1j * w.cpu().numpy()
        V = skewgpu.from_device(x) + 1j * skewgpu.from_device(y)
        # n reflectors and about 2 n rotations of a row, each orthogonal to a few eps
        assert np.linalg.norm(V.conj().T @ V - np.eye(n), 2) <= 20 * n * EPS
        assert np.linalg.norm(A @ V - V * lam, 2) <= 20 * n * EPS * max(np.linalg.norm(A, 2), 1.0)
    plan.close()
