"""Coupled operands of very different size.  The tensor-core products and the large reductions hold their
operands in 56 bits relative to the largest entry of a row, column or tile, so their errors are those of
Float64 arithmetic relative to these entries: bounded by n eps times the norm of the whole, and not, as
entry by entry in Float64, relative to each small block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sl = pytest.importorskip("scipy.linalg")

EPS = np.finfo(float).eps


def _skew(n, seed):
    B = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    return B - B.T


@pytest.mark.parametrize("ratio", [1e-3, 1e-6, 1e-9])
def test_adjoint_of_a_graded_cotangent(skewgpu, ratio):
    m, n = 70, 140
    A = np.zeros((n, n))
    A[:m, :m], A[m:, m:] = _skew(m, 1), _skew(m, 2)
    d = np.where(np.arange(n) < m, 1.0, ratio)
    C = d[:, None] * np.random.default_rng(3).standard_normal((n, n)) * d
    _, pullback = skewgpu.exp_rrule(A)
    G = pullback(C)
    for i in (0, m):  # block (i, j) of the result depends on that block of C alone
        for j in (0, m):
            si, sj = slice(i, i + m), slice(j, j + m)
            M = np.zeros((2 * m, 2 * m))
            M[:m, :m], M[m:, m:], M[:m, m:] = A[si, si].T, A[sj, sj].T, C[si, sj]
            want = sl.expm(M)[:m, m:] if i != j else sl.expm_frechet(A[si, si].T, C[si, sj], compute_expm=False)
            assert np.linalg.norm(G[si, sj] - want) <= 40 * n * EPS * np.linalg.norm(C)


@pytest.mark.parametrize("n,decades", [(700, 6), (700, 12), (1100, 8)])
def test_reduction_of_a_graded_matrix(skewgpu, n, decades):
    d = 10.0 ** (-decades * np.arange(n) / n)
    A = np.tril(d[:, None] * _skew(n, n) * d)
    A -= A.T  # skew to the last bit
    H = skewgpu.hessenberg(A)
    ev = H.ev.cpu().numpy()
    got = np.linalg.svd(np.diag(ev, 1) - np.diag(ev, -1), compute_uv=False)
    want = np.linalg.svd(A, compute_uv=False)
    # Weyl: singular values move by no more than the backward error, a modest multiple of sqrt(n) eps |A|
    assert np.abs(got - want).max() <= 32 * np.sqrt(n) * EPS * want[0]
