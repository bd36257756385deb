"""exp, cis, functions and the exp adjoint of one real matrix whose tridiagonal splits into more
odd blocks than n mod 2 (zero padding, blocks of odd size, the zero matrix): the eigenvectors come
from the full mode, whose back-transformation takes 2 n columns.  On a handle of its own, so the
workspace is no larger than the call asks for."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
sl = pytest.importorskip("scipy.linalg")

EPS = np.finfo(float).eps


def _matrix(kind, n):
    A = np.zeros((n, n))
    rng = np.random.default_rng(n)

    def fill(o, m):
        B = rng.standard_normal((m, m)) / np.sqrt(m)
        A[o:o + m, o:o + m] = B - B.T

    if kind == "padded":
        fill(0, n - 2 - n % 2)
    elif kind == "blocks":
        m = (n // 2) | 1
        fill(0, m)
        fill(m, n - m)
    return A


@pytest.mark.parametrize("kind", ["padded", "blocks", "zero"])
@pytest.mark.parametrize("n", [96, 108, 112, 128, 130, 160, 192])
def test_functions(skewgpu, kind, n):
    import torch
    from skewgpu import _lib
    from skewgpu._lib import check

    A = _matrix(kind, n)
    C = np.random.default_rng(n + 1).standard_normal((n, n))
    L = _lib.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    info = torch.full((1,), -1, dtype=torch.int32, device="cuda")

    def call(f, out, *extra):
        h = ctypes.c_void_p()
        check(L.skew_create(ctypes.byref(h)))
        check(L.skew_set_stream(h, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        W = skewgpu.to_device(A)
        check(f(h, p(W), n, n, *extra, p(out), n, p(info)))
        assert int(info.item()) == 0
        check(L.skew_destroy(h))
        return out.cpu().numpy().T  # column-major

    new = lambda t: torch.zeros((n, n), dtype=t, device="cuda")  # noqa: E731
    # n-th order eigenproblem and products of orthogonal matrices: a modest multiple of n eps |f|
    tol = 40 * n * EPS
    want = sl.expm(A)
    assert np.linalg.norm(call(L.skew_exp_d, new(torch.float64)) - want) <= tol * np.linalg.norm(want)
    want = sl.expm(1j * A)
    assert np.linalg.norm(call(L.skew_cis_d, new(torch.complex128)) - want) <= tol * np.linalg.norm(want)
    want = sl.sinm(A)
    got = call(lambda h, a, n_, l, o, lo, i: L.skew_func_d(h, a, n_, l, 2, o, lo, i), new(torch.float64))
    assert np.linalg.norm(got - want) <= tol * max(np.linalg.norm(want), np.linalg.norm(A))
    # G = d<C, exp(A)>: the Frechet derivative of exp at A^T in direction C
    want = sl.expm_frechet(A.T, C, compute_expm=False)
    dC = skewgpu.to_device(C)
    got = call(lambda h, a, n_, l, o, lo, i: L.skew_exp_vjp_d(h, a, n_, l, p(dC), o, lo, i), new(torch.float64))
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
