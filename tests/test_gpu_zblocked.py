"""The blocked complex reduction of one matrix: threads per row and matvec chunks over grid
sizes, ragged panels, and its indifference to powers of two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def skewh(n, seed):
    rng = np.random.default_rng(seed)
    C = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (C - C.conj().T) / 2


def form_q(F, tau):
    n = F.shape[0]
    Q = np.eye(n, dtype=complex)
    for j in range(len(tau) - 1, -1, -1):
        v = F[j + 1:, j].copy()
        v[0] = 1.0
        Q[j + 1:, j + 1:] -= tau[j] * np.outer(v, v.conj() @ Q[j + 1:, j + 1:])
    return Q


# grid of g CTAs: 32, 16, 8, 4 threads per row while at most 4 g, 8 g, 16 g, more rows are left
@pytest.mark.parametrize("n,ctas,nb", [(131, 0, 32), (193, 2, 32), (260, 3, 5), (400, 40, 32), (545, 24, 31),
                                       (640, 0, 32), (737, 0, 32)])
def test_reduction(skewgpu, n, ctas, nb):
    A = skewh(n, n)
    with skewgpu.tuned(zpersist_min_n=130, zpersist_ctas=ctas, zpersist_nb=nb):
        H = skewgpu.hessenberg_complex(A)
    tau = H.tau.cpu().numpy()
    Q = form_q(skewgpu.from_device_complex(H.factors), tau)
    eps = np.finfo(float).eps
    # n reflectors, each orthogonal and applied to a few rounding errors: 10 n eps
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(n), 2) <= 10 * n * eps
    assert np.linalg.norm(Q.conj().T @ A @ Q - H.H()) <= 10 * n * eps * np.linalg.norm(A)


@pytest.mark.parametrize("k", [-400, 300])
def test_power_of_two(skewgpu, k):
    """Every operation of the panels is homogeneous: the scaled matrix gives the same bits."""
    n = 450
    A = skewh(n, 7)
    a, b = skewgpu.hessenberg_complex(A), skewgpu.hessenberg_complex(np.ldexp(A.real, k) + 1j * np.ldexp(A.imag, k))
    m = n - 129
    np.testing.assert_array_equal(b.tau.cpu().numpy()[:m], a.tau.cpu().numpy()[:m])
    np.testing.assert_array_equal(b.ev.cpu().numpy()[:m], np.ldexp(a.ev.cpu().numpy()[:m], k))


def test_zero_columns(skewgpu):
    """Columns without a reflector inside a panel: the identity there, zeros beside it."""
    n, z = 420, 40
    A = skewh(n, 9)
    A[:z, :] = 0.0
    A[:, :z] = 0.0
    H = skewgpu.hessenberg_complex(A)
    np.testing.assert_array_equal(H.ev.cpu().numpy()[:z], 0.0)
    np.testing.assert_array_equal(H.tau.cpu().numpy()[: z - 1], 0.0)
    Q = form_q(skewgpu.from_device_complex(H.factors), H.tau.cpu().numpy())
    assert np.linalg.norm(Q.conj().T @ A @ Q - H.H()) <= 10 * n * np.finfo(float).eps * np.linalg.norm(A)
