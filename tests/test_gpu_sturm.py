"""Eigenvalues by Sturm counts of the leading blocks' polynomials: sizes from the smallest
to past the rows a CTA stages, splits, tiny and graded couplings, extreme scales."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _symtri_abs(e):
    """|eigenvalues| of SymTridiagonal(0, e), descending (LAPACK's bisection)."""
    from scipy.linalg import eigvalsh_tridiagonal

    n = len(e) + 1
    s = np.abs(e).max() if n > 1 and np.abs(e).max() > 0 else 1.0
    w = eigvalsh_tridiagonal(np.zeros(n), np.abs(e) / s, lapack_driver="stebz")
    return np.sort(np.abs(w))[::-1] * s


def _svdvals(e):
    """By bisection at every size: dense up to n = 1024 (where the tridiagonal entry runs the QR;
    reducing a tridiagonal matrix only flips signs), tridiagonal above."""
    import skewgpu

    n = len(e) + 1
    if n > 1024:
        return skewgpu.SkewHermTridiagonal(e).svdvals()
    T = np.zeros((n, n))
    T[np.arange(1, n), np.arange(n - 1)] = e
    T[np.arange(n - 1), np.arange(1, n)] = -e
    return skewgpu.svdvals(T)


CASES = [(n, kind) for n in (2, 3, 33, 64, 257, 1025) for kind in ("normal", "split", "graded", "huge", "small")]
CASES += [(n, "normal") for n in (3072, 3073)]


@pytest.mark.parametrize("n,kind", CASES)
def test_svdvals_of_tridiagonal(n, kind):
    rng = np.random.default_rng(100 * n + len(kind))
    e = rng.standard_normal(n - 1)
    if kind == "split":
        e[:: max(2, n // 7)] = 0.0
    elif kind == "graded":
        e *= 2.0 ** (-1.0 * (np.arange(n - 1) % 40))
    elif kind == "huge":
        e *= 1e150
    elif kind == "small":
        e *= 1e-150
    got = _svdvals(e)
    want = _symtri_abs(e)
    # both bracket within a few eps of the norm; a count errs by a few eps of the entries per row;
    # the search stops at brackets of 4 x the smallest normal number (a zero matrix)
    assert np.abs(got - want).max() <= 16 * EPS * max(want.max(), np.abs(e).max()) + 4 * np.finfo(float).tiny


@pytest.mark.parametrize("n", [2, 65, 1024, 3073])
def test_complex_tridiagonal_with_diagonal(n):
    import skewgpu
    from scipy.linalg import eigvalsh_tridiagonal

    rng = np.random.default_rng(n)
    ev = rng.standard_normal(n - 1) + 1j * rng.standard_normal(n - 1)
    d = rng.standard_normal(n)
    d[n // 2] = 0.0
    ev[n // 3] = 0.0
    got = skewgpu.SkewHermTridiagonal(ev, d).eigvals().imag
    want = np.sort(-eigvalsh_tridiagonal(-d, np.abs(ev), lapack_driver="stebz"))[::-1]
    assert np.abs(np.sort(got)[::-1] - want).max() <= 16 * EPS * (np.abs(d).max() + 2 * np.abs(ev).max())


def test_tiny_singular_value_keeps_relative_accuracy():
    # couplings (a, b, a) give singular values of [[a, 0], [b, a]]: s1 s2 = a^2, s1^2 + s2^2 = 2 a^2 + b^2
    a, b = 1e-9, 1.0
    got = _svdvals(np.array([a, b, a]))
    s1 = np.sqrt((2 * a * a + b * b + b * np.sqrt(4 * a * a + b * b)) / 2)
    s2 = a * a / s1
    assert abs(got.min() - s2) <= 16 * EPS * s2 and abs(got.max() - s1) <= 16 * EPS * s1
