"""The trailing updates of the large reductions on the tensor cores (real n > 640, complex n >= 384)
at matrix scales whose square leaves the double range, and the real one's smallest sizes."""
import numpy as np
import pytest

from test_gpu_wide import _check, _reduce, _skew
from test_gpu_zblocked import skewh

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [641, 642, 671, 705])
def test_smallest_sizes(n):
    A = _skew(n, n)
    _check(A, *_reduce(A))


@pytest.mark.parametrize("n", [650, 1100])
@pytest.mark.parametrize("k", [-515, 515, 900])
def test_real(n, k):
    """2^k A has the reflectors of A and 2^k times its subdiagonal."""
    A = _skew(n, 5)
    T0, tau0, ev0 = _reduce(A)
    T1, tau1, ev1 = _reduce(np.ldexp(A, k))
    # every step is homogeneous, but the norms of very large or small columns are formed from
    # scaled entries: their rounding, amplified as any rounding of the reduction is
    assert np.abs(np.ldexp(ev1, -k) - ev0).max() <= 1e-11 * np.abs(ev0).max()
    assert np.abs(tau1 - tau0).max() <= 1e-11
    _check(A, T1, tau1, np.ldexp(ev1, -k))


@pytest.mark.parametrize("k", [-505, 530, 900])
def test_complex(skewgpu, k):
    n = 450
    A = skewh(n, 7)
    a, b = skewgpu.hessenberg_complex(A), skewgpu.hessenberg_complex(np.ldexp(A.real, k) + 1j * np.ldexp(A.imag, k))
    ev0, ev1 = a.ev.cpu().numpy(), np.ldexp(b.ev.cpu().numpy(), -k)
    assert np.abs(ev1 - ev0).max() <= 1e-11 * np.abs(ev0).max()
    assert np.abs(b.tau.cpu().numpy() - a.tau.cpu().numpy()).max() <= 1e-11
