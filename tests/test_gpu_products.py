"""The tensor-core products behind exp, cis and the exp adjoint: sizes at the edges of the
128 x 64 tiles, of the 32-entry buffers and of the 128-entry exact sums, rows of very
different scales, and entries that are not finite."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [4, 15, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 160, 192, 255, 257]
EPS = np.finfo(float).eps


def _batch(sizes, seed, radius=3.0):
    rng = np.random.default_rng(seed)
    mats = []
    for n in sizes:
        B = rng.standard_normal((n, n))
        mats.append((B - B.T) / 2 * radius / np.sqrt(2.0 * n))
    return mats, rng


def _frechet(A, C):
    import scipy.linalg as sl

    n = len(A)
    M = np.zeros((2 * n, 2 * n))
    M[:n, :n] = M[n:, n:] = A.T
    M[:n, n:] = C
    return sl.expm(M)[:n, n:]


def _run_vjp(mats, cots):
    import skewgpu

    dA = [skewgpu.to_device(A) for A in mats]
    dC = [skewgpu.to_device(C) for C in cots]
    dG = [torch.zeros_like(a) for a in dA]
    plan = skewgpu.BatchPlan([len(A) for A in mats])
    st = plan.exp_vjp(plan.pointer_array(dA), plan.pointer_array(dC), plan.pointer_array(dG))
    out = [skewgpu.from_device(G) for G in dG]
    plan.close()
    return out, st.cpu().numpy()


def test_exp_vjp_at_tile_edges():
    mats, rng = _batch(SIZES, 1)
    cots = [rng.standard_normal(A.shape) for A in mats]
    got, st = _run_vjp(mats, cots)
    assert (st == 0).all()
    for A, C, G in zip(mats, cots, got):
        want = _frechet(A, C)
        # eigenpairs and four products: a modest multiple of n eps, norm-wise
        assert np.linalg.norm(G - want) <= 40 * max(len(A), 32) * EPS * np.linalg.norm(want), len(A)


@pytest.mark.parametrize("schur", [1, 0])
def test_cis_both_forms_at_tile_edges(schur):
    import scipy.linalg as sl
    import skewgpu

    mats, _ = _batch(SIZES, 2)
    with skewgpu.tuned(func_real_schur=schur):
        dA = [skewgpu.to_device(A) for A in mats]
        dC = [torch.zeros((len(A), len(A), 2), dtype=torch.float64, device="cuda") for A in mats]
        plan = skewgpu.BatchPlan(SIZES)
        plan.cis(plan.pointer_array(dA), plan.pointer_array(dC))
        got = [(c.cpu().numpy()[..., 0] + 1j * c.cpu().numpy()[..., 1]).T for c in dC]
        plan.close()
    for A, G in zip(mats, got):
        want = sl.expm(1j * A)
        assert np.linalg.norm(G - want) <= 40 * max(len(A), 32) * EPS * np.linalg.norm(want), len(A)


def test_blocks_of_different_scale_keep_their_accuracy():
    """A block-diagonal A and a cotangent 1e12 times larger on one block: the rows and columns of the
    products have their own scales, so the small block's gradient is as accurate as alone."""
    (A1, A2), rng = _batch([48, 80], 3)
    n1, n = 48, 128
    A = np.zeros((n, n))
    A[:n1, :n1], A[n1:, n1:] = A1, A2
    C = np.zeros((n, n))
    C[:n1, :n1] = 1e12 * rng.standard_normal((n1, n1))
    C[n1:, n1:] = rng.standard_normal((n - n1, n - n1))
    (G,), _ = _run_vjp([A], [C])
    for s in (slice(0, n1), slice(n1, n)):
        want = _frechet(A[s, s], C[s, s])
        assert np.linalg.norm(G[s, s] - want) <= 40 * n * EPS * np.linalg.norm(want)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite_cotangent_gives_nan(bad):
    mats, rng = _batch([70, 70], 4)
    cots = [rng.standard_normal(A.shape) for A in mats]
    cots[0][3, 5] = bad
    (G0, G1), _ = _run_vjp(mats, cots)
    assert np.isnan(G0).all()
    want = _frechet(mats[1], cots[1])
    assert np.linalg.norm(G1 - want) <= 40 * 70 * EPS * np.linalg.norm(want)


@pytest.mark.parametrize("n", [95, 96, 97, 160, 333, 640, 641, 700, 1024])
def test_single_matrix_functions_at_the_dispatch_edges(n):
    """exp and its adjoint of one matrix around the sizes where the whole GPU takes over (96) and
    where its reduction changes (641)."""
    import scipy.linalg as sl
    import skewgpu

    (A,), rng = _batch([n], 10 + n)
    want = sl.expm(A)
    assert np.linalg.norm(skewgpu.exp(A) - want) <= 40 * n * EPS * np.linalg.norm(want)
    if n <= 333:
        C = rng.standard_normal((n, n))
        _, pullback = skewgpu.exp_rrule(A)
        ref = _frechet(A, C)
        assert np.linalg.norm(pullback(C) - ref) <= 40 * n * EPS * np.linalg.norm(ref)
    if n % 2:
        with pytest.raises(ValueError):
            skewgpu.matrix_function(A, "log")
