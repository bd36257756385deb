"""The reduction of one real matrix above n = 1024 (panel products in fixed point, trailing
update on the tensor cores): sizes at the edges of the 64-row tiles, the last partial panel
and the tail, panel widths, splits, extreme scales and rows of very different size."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _skew(n, seed):
    B = np.random.default_rng(seed).standard_normal((n, n))
    return (B - B.T) / 2


def _reduce(A):
    import skewgpu

    F = skewgpu.hessenberg(A)
    T = F.factors.cpu().numpy()  # T[j, i] = A[i, j]: rows are columns of the reduced matrix
    return T, F.tau.cpu().numpy(), F.ev.cpu().numpy()


def _residual(A, T, tau, ev):
    """|Q H Q^T - A| and |Q^T Q - I| with Q applied reflector by reflector (torch, FP64, on the GPU)."""
    n = len(A)
    Q = torch.eye(n, dtype=torch.float64, device="cuda")
    dT = torch.from_numpy(T).cuda()
    for c in range(n - 2, -1, -1):
        if tau[c] == 0.0:
            continue
        v = dT[c].clone()
        v[: c + 1] = 0.0
        v[c + 1] = 1.0
        Q -= tau[c] * torch.outer(v, v @ Q)
    H = torch.zeros_like(Q)
    e = torch.from_numpy(ev).cuda()
    i = torch.arange(n - 1, device="cuda")
    H[i + 1, i], H[i, i + 1] = e, -e
    dA = torch.from_numpy(A).cuda()
    return (float(torch.linalg.norm(Q @ H @ Q.T - dA)),
            float(torch.linalg.norm(Q.T @ Q - torch.eye(n, dtype=torch.float64, device="cuda"))))


def _check(A, T, tau, ev):
    n = len(A)
    norm = np.linalg.norm(A)
    r, o = _residual(A / norm if norm else A, T, tau, ev / norm if norm else ev)
    # norm-wise backward error of n two-sided reflections (a few n^(1/2) eps each way in practice)
    assert r <= 4 * np.sqrt(n) * EPS * 8 and o <= 4 * n * EPS


@pytest.mark.parametrize("n", [1025, 1088, 1089, 1090, 1152, 1153, 1217, 1281, 1500])
def test_sizes_at_tile_and_panel_edges(n):
    A = _skew(n, n)
    T, tau, ev = _reduce(A)
    _check(A, T, tau, ev)


def test_against_oracle():
    from oracle import oracle as O

    n = 1100
    A = _skew(n, 7) / np.sqrt(n)
    _, tq, evq = O.hessenberg(A)
    T, tau, ev = _reduce(A)
    assert np.abs(ev - evq).max() <= 1e-11 * np.abs(evq).max()
    assert np.array_equal(tau != 0, tq != 0)


@pytest.mark.parametrize("keys", [dict(persist_nb=8), dict(persist_nb=40), dict(persist_ctas=37),
                                  dict(persist_tail=33)])
def test_tuning_keys(keys):
    import skewgpu

    A = _skew(1200, 3)
    with skewgpu.tuned(**keys):
        T, tau, ev = _reduce(A)
    _check(A, T, tau, ev)


@pytest.mark.parametrize("s", [1e150, 1e-150])
def test_scale_invariance(s):
    """A power of two times A: the same reflectors bit for bit, ev scaled."""
    A = _skew(1100, 5)
    f = 2.0 ** np.round(np.log2(s))
    T0, tau0, ev0 = _reduce(A)
    T1, tau1, ev1 = _reduce(A * f)
    # the norms of very large or small columns are formed from scaled entries
    assert np.abs(ev1 / f - ev0).max() <= 1e-12 * np.abs(ev0).max()
    assert np.abs(tau1 - tau0).max() <= 1e-12


def test_zero_and_split_matrices():
    n = 1200
    T, tau, ev = _reduce(np.zeros((n, n)))
    assert not ev.any() and not tau.any()
    A = np.zeros((n, n))
    A[:500, :500], A[500:, 500:] = _skew(500, 8), _skew(700, 9)
    T, tau, ev = _reduce(A)
    _check(A, T, tau, ev)


def test_blocks_of_different_scale():
    """Two uncoupled blocks 1e12 apart: tiles and vectors have their own scales, so the small
    block is reduced as accurately as alone."""
    n, m = 1216, 640
    A = np.zeros((n, n))
    A[:m, :m] = 1e12 * _skew(m, 10)
    A[m:, m:] = _skew(n - m, 11)
    _, _, ev = _reduce(A)
    w = np.linalg.eigvalsh(1j * A[m:, m:])
    H = np.diag(1j * ev[m:], 1)
    got = np.linalg.eigvalsh(H + H.conj().T)
    assert np.abs(np.sort(np.abs(got)) - np.sort(np.abs(w))).max() <= 1e-12 * np.abs(w).max()


def test_not_finite_entries_reach_the_result():
    A = _skew(1100, 12)
    A[700, 300] = np.nan
    A[300, 700] = np.nan
    import skewgpu

    F = skewgpu.hessenberg(skewgpu.SkewHermitian(skewgpu.to_device(A), check_skew=False))
    assert np.isnan(F.ev.cpu().numpy()).any()


def test_timeout_is_reported_and_leaves_the_next_call_sound():
    import skewgpu
    from skewgpu import _lib

    A = _skew(1100, 13)
    L, h = _lib.load(), skewgpu.handle().bind()
    n = len(A)

    def call():
        import ctypes

        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        W = skewgpu.to_device(A)
        tau = torch.zeros(n - 1, dtype=torch.float64, device="cuda")
        ev = torch.zeros_like(tau)
        info = torch.zeros(1, dtype=torch.int32, device="cuda")
        assert L.skew_hessenberg_d(h, p(W), n, n, p(tau), p(ev), p(info)) == 0
        return int(info.item()), ev.cpu().numpy()

    ok, ev0 = call()
    with skewgpu.tuned(wait_polls=20000, wait_skip_cta=3):
        bad, _ = call()
    again, ev1 = call()
    assert ok == 0 and bad == _lib.SKEW_TIMEOUT and again == 0
    assert np.array_equal(ev0, ev1)
