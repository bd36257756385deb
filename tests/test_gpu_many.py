"""Batches of more matrices than a grid counts in y or z (65 535)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _pointers(buf, n, index):
    base = buf.data_ptr() + 8 * n * n * np.asarray(index, dtype=np.int64)
    return torch.tensor(base.tolist(), dtype=torch.int64, device="cuda")


def test_gradients(skewgpu):
    """65 600 matrices above n = 96, 50 different ones: each has the gradient of its first occurrence."""
    count, n, kinds = 65600, 98, 50
    rng = np.random.default_rng(1)
    B = rng.standard_normal((kinds, n, n)) / np.sqrt(n)
    A = (B - B.transpose(0, 2, 1)) / 2
    k = np.arange(0, n, 2)
    A[:, k, k + 1] += 2.0
    A[:, k + 1, k] -= 2.0
    dA = torch.from_numpy(np.ascontiguousarray(A.transpose(0, 2, 1))).cuda()
    G = torch.zeros((count, n, n), dtype=torch.float64, device="cuda")
    out = [torch.zeros(count, dtype=torch.float64, device="cuda") for _ in range(2)]
    st = torch.full((count,), -1, dtype=torch.int32, device="cuda")
    plan = skewgpu.BatchPlan([n] * count)
    plan.logabspfaffian(_pointers(dA, n, np.arange(count) % kinds), _pointers(G, n, np.arange(count)), *out, st)
    torch.cuda.synchronize()
    assert not st.any()
    want = np.linalg.inv(A).transpose(0, 2, 1) / 2
    first = G[:kinds].cpu().numpy().transpose(0, 2, 1)
    for b in range(kinds):  # well-conditioned: a modest multiple of n eps
        assert np.linalg.norm(first[b] - want[b]) <= 20 * n * EPS * np.linalg.norm(want[b])
    for b in range(0, count, kinds):
        assert torch.equal(G[b:b + kinds], G[:kinds])
    plan.close()


def test_eigen(skewgpu):
    """70 000 small matrices and one whose back-transformation runs on the tensor cores."""
    count, n, big = 70000, 3, 48
    rng = np.random.default_rng(2)
    B = rng.standard_normal((n, n))
    C = rng.standard_normal((big, big))
    mats = [(B - B.T) / 2, (C - C.T) / 2]
    sizes = [n] * count + [big]
    small, large = skewgpu.to_device(mats[0]), skewgpu.to_device(mats[1])
    V = [torch.zeros(n * n * count + big * big, dtype=torch.float64, device="cuda") for _ in range(2)]
    vals = torch.zeros(n * count + big, dtype=torch.float64, device="cuda")
    pA = torch.tensor([small.data_ptr()] * count + [large.data_ptr()], dtype=torch.int64, device="cuda")
    at = np.append(np.arange(count), count)
    pv = torch.tensor((vals.data_ptr() + 8 * n * at).tolist(), dtype=torch.int64, device="cuda")
    st = torch.full((count + 1,), -1, dtype=torch.int32, device="cuda")
    plan = skewgpu.BatchPlan(sizes)
    plan.eigen(pA, pv, _pointers(V[0], n, at), _pointers(V[1], n, at), st)
    torch.cuda.synchronize()
    assert not st.any()
    lam = 1j * vals.cpu().numpy()
    W = V[0].cpu().numpy() + 1j * V[1].cpu().numpy()
    for b in (0, 65534, 65535, 65536, count - 1, count):
        m = big if b == count else n
        A = mats[b == count]
        v, w = lam[n * b:n * b + m], W[n * n * b:n * n * b + m * m].reshape(m, m).T
        assert np.linalg.norm(A @ w - w * v) <= 40 * m * EPS * np.linalg.norm(A)
        assert np.linalg.norm(w.conj().T @ w - np.eye(m)) <= 40 * m * EPS
    plan.close()
