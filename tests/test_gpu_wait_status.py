"""A bounded wait that gives up in a back-transformation is reported: one CTA's tiles count as given
up (tuning key wait_skip_cta; nothing waits, nothing is in flight), and the call's status says so."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _skewh(n, seed):
    rng = np.random.default_rng(seed)
    C = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (C - C.conj().T) / 2


def test_functions_of_one_real_matrix(skewgpu):
    A = _skewh(200, 1).real / 10  # one cluster reduces it: the back-transformation's waits alone
    good = skewgpu.exp(A)
    with skewgpu.tuned(wait_skip_cta=0):
        with pytest.raises(skewgpu.SkewError):
            skewgpu.exp(A)
    np.testing.assert_array_equal(skewgpu.exp(A), good)


def test_eigen_of_one_complex_matrix(skewgpu):
    A = _skewh(100, 2)
    good = skewgpu.eigen_complex(A)[0]
    with skewgpu.tuned(wait_skip_cta=0):
        with pytest.raises(skewgpu.SkewError):
            skewgpu.eigen_complex(A)
    np.testing.assert_array_equal(skewgpu.eigen_complex(A)[0], good)


def test_batched_complex_status(skewgpu):
    n, count = 70, 3
    A = torch.stack([skewgpu.to_device_complex(_skewh(n, k) / 10) for k in range(count)])
    E = torch.zeros_like(A)
    L, h = skewgpu._lib.load(), skewgpu.handle().bind()
    status = torch.full((count,), -1, dtype=torch.int32, device="cuda")

    def call():
        assert L.skew_batch_exp_z(h, _p(A), n, count, _p(E), _p(status)) == 0
        return status.cpu().tolist()

    assert call() == [0] * count
    with skewgpu.tuned(wait_skip_cta=0):
        assert call() == [skewgpu._lib.SKEW_TIMEOUT] * count
    assert call() == [0] * count


# the wide reduction, and without the cluster one the grid-wide one
@pytest.mark.parametrize("n,keys", [(1100, {}), (512, dict(cluster_max_n=0))])
def test_logabspf_keeps_the_reductions_timeout(skewgpu, n, keys):
    A = _skewh(n, n).real / np.sqrt(n)
    L, h = skewgpu._lib.load(), skewgpu.handle().bind()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    info = torch.full((1,), -1, dtype=torch.int32, device="cuda")

    def call():
        W = skewgpu.to_device(A)
        assert L.skew_logabspf_d(h, _p(W), n, n, _p(out), ctypes.c_void_p(out.data_ptr() + 8), 0, _p(info)) == 0
        return int(info.item()), out.cpu().numpy()

    ok, good = call()
    with skewgpu.tuned(wait_polls=20000, wait_skip_cta=3, **keys):
        bad, nans = call()
        with pytest.raises(skewgpu.SkewError):
            skewgpu.logabspfaffian(A)
    again, after = call()
    assert (ok, bad, again) == (0, skewgpu._lib.SKEW_TIMEOUT, 0)
    assert np.isnan(nans).all()
    np.testing.assert_array_equal(good, after)
