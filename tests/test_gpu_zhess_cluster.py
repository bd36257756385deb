"""The batched complex reduction at every cluster width (1, 2, 4 and 8 CTAs per matrix), sizes
at the edges of its 32-row blocks, matrices that decouple, and the tail of larger ones."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _mats(count, n, seed):
    rng = np.random.default_rng(seed)
    C = rng.standard_normal((count, n, n)) + 1j * rng.standard_normal((count, n, n))
    return (C - C.conj().transpose(0, 2, 1)) / 2


@pytest.mark.parametrize("count,n", [(200, 33), (200, 65), (100, 130), (40, 127), (40, 257), (3, 64), (3, 129),
                                     (2, 320), (2, 511), (2, 512), (5, 1), (5, 2), (5, 3)])
def test_batched_eigen(count, n):
    import skewgpu

    A = _mats(count, n, 10 * n + count)
    vals, V = skewgpu.batch_eigen_complex(list(A))
    for k in range(0, count, max(1, count // 6)):
        v, lam = V[k], vals[k]
        norm = max(np.linalg.norm(A[k]), 1e-300)
        assert np.linalg.norm(A[k] @ v - v * lam) <= 16 * np.sqrt(n) * EPS * norm
        assert np.linalg.norm(v.conj().T @ v - np.eye(n)) <= 8 * n * EPS
        want = np.sort(np.linalg.eigvalsh(1j * A[k]))
        assert np.abs(np.sort(-lam.imag) - want).max() <= 16 * np.sqrt(n) * EPS * np.abs(want).max()


def test_decoupled_columns():
    """Zero columns (reflectors that are the identity) in a batch on clusters of 4 and 8."""
    import skewgpu

    for count, n in ((40, 256), (2, 512)):
        A = _mats(count, n, n)
        h = n // 2
        A[:, :h, h:] = 0.0
        A[:, h:, :h] = 0.0
        A[0] = np.diag(1j * np.arange(n))
        vals, V = skewgpu.batch_eigen_complex(list(A))
        for k in (0, 1):
            assert np.linalg.norm(A[k] @ V[k] - V[k] * vals[k]) <= 16 * np.sqrt(n) * EPS * np.linalg.norm(A[k])
            assert np.linalg.norm(V[k].conj().T @ V[k] - np.eye(n)) <= 8 * n * EPS
