"""Eigenvalues by counts and interpolation: 32, 16, 8, 4, 2 and 1 lanes per eigenvalue, spectra
known in closed form, simple, close and multiple."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def block(rng, m):
    e = rng.standard_normal(m - 1)
    T = np.diag(e, 1) + np.diag(e, -1)
    return e, np.abs(np.linalg.eigvalsh(T))


@pytest.mark.parametrize("n", [1101, 1300, 4500, 5001, 12000, 20001])
@pytest.mark.parametrize("kind", ["ones", "multiple", "close", "far"])
def test_svdvals_known(skewgpu, n, kind):
    rng = np.random.default_rng(n)
    if kind == "ones":
        e = np.ones(n - 1)
        want = np.abs(2.0 * np.cos(np.arange(1, n + 1) * np.pi / (n + 1)))
    else:
        m = 20
        b, w = block(rng, m)
        reps = n // m
        f = np.ones(reps)
        if kind == "close":  # neighbours 1e-10 apart
            f += 1e-10 * np.arange(reps)
        elif kind == "far":  # 200 binary orders
            f = 2.0 ** np.linspace(-200.0, 0.0, reps).round()
        e = np.zeros(n - 1)
        want = np.zeros(n)
        for r in range(reps):
            e[r * m:r * m + m - 1] = f[r] * b
            want[r * m:(r + 1) * m] = f[r] * w
    got = skewgpu.SkewHermTridiagonal(e).svdvals()
    want = np.sort(want)[::-1]
    # brackets of 2 eps; a count errs by a few eps of the entries per row; the blocks' own error
    assert np.abs(got - want).max() <= 32 * EPS * want.max()
