"""A NaN or an infinity in a large matrix is not lost between the panels of its reduction."""
import numpy as np
import pytest

from test_gpu_wide import _skew

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e3])
def test_hessenberg(skewgpu, bad, scale):
    n = 1000
    A = scale * _skew(n, 12)
    A[700, 300], A[300, 700] = bad, -bad
    ev = skewgpu.hessenberg(skewgpu.SkewHermitian(skewgpu.to_device(A), check_skew=False)).ev.cpu().numpy()
    # the first column's product spreads it over the rows, the second's norm over all that follow
    assert np.isfinite(ev[0]) and not np.isfinite(ev[1:]).any()
