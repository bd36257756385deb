"""The cluster reduction of complex matrices writes into its CTAs' shared memory from the first
column on, so it starts with a barrier of the cluster: many clusters at once, and waiting ones,
give the same bits every time."""
import numpy as np
import pytest

from test_gpu_zhess_cluster import _mats

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,n", [(150, 130), (75, 256), (2, 512)])  # clusters of 2, 4 and 8
def test_same_bits_on_every_run(skewgpu, count, n):
    A = list(_mats(count, n, n))
    first = skewgpu.batch_eigen_complex(A)
    for _ in range(5):
        again = skewgpu.batch_eigen_complex(A)
        for x, y in zip(first, again):
            np.testing.assert_array_equal(np.asarray(x), np.asarray(y))
    lam, v = first[0][0], first[1][0]
    assert np.linalg.norm(A[0] @ v - v * lam) <= 16 * np.sqrt(n) * np.finfo(float).eps * np.linalg.norm(A[0])
