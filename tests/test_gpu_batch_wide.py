"""Batched reductions with 16 warps per matrix (batches whose largest matrix sets the time, and
sizes from 384 on): exp against dense linear algebra."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def skew(n, seed):
    B = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    A = (B - B.T) / 2
    k = np.arange(0, n - 1, 2)
    A[k, k + 1] += 2.0
    A[k + 1, k] -= 2.0
    return A


BATCHES = [[97], [98, 16, 33], [128, 383], [384, 384], [511, 512, 100, 31], [256] + [100] * 20]


@pytest.mark.parametrize("sizes", BATCHES, ids=lambda s: "-".join(map(str, s[:4])))
def test_batch(skewgpu, sizes):
    mats = [skew(n, n + i) for i, n in enumerate(sizes)]
    dA = [skewgpu.to_device(A) for A in mats]
    plan = skewgpu.BatchPlan(sizes)
    dO = [torch.zeros_like(a) for a in dA]
    plan.exp(plan.pointer_array(dA), plan.pointer_array(dO))
    for A, O in zip(mats, dO):
        n = len(A)
        w, V = np.linalg.eigh(1j * A)
        want = ((V * np.exp(-1j * w)) @ V.conj().T).real
        # eigenvectors orthogonal to a few n eps, products of norm 1
        assert np.linalg.norm(skewgpu.from_device(O) - want, 2) <= 20 * n * EPS
    plan.close()
