"""Gradients of the batched log|Pf| on the tensor cores (matrices above the shared-memory
sizes): sizes at the edges of tiles and panels, odd and singular matrices among them, a
replayed plan, new contents behind the same pointers, and badly conditioned matrices."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _skew(n, seed, j=0.0):
    B = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    A = (B - B.T) / 2
    k = np.arange(0, n - 1, 2)
    A[k, k + 1] += j
    A[k + 1, k] -= j
    return A


def _run(mats, plan=None):
    import skewgpu

    dA = [skewgpu.to_device(A) for A in mats]
    dG = [torch.full_like(a, 7.0) for a in dA]
    own = plan is None
    plan = plan or skewgpu.BatchPlan([len(A) for A in mats])
    lp, sg, st = plan.logabspfaffian(plan.pointer_array(dA), plan.pointer_array(dG))
    out = [skewgpu.from_device(G) for G in dG], lp.cpu().numpy(), sg.cpu().numpy(), st.cpu().numpy()
    if own:
        plan.close()
    return out


SIZES = [98, 100, 126, 128, 130, 132, 160, 190, 192, 194, 254, 256, 258, 260, 384, 390, 512]


def test_sizes_at_tile_and_panel_edges():
    mats = [_skew(n, n, 2.0) for n in SIZES]
    G, lp, sg, st = _run(mats)
    assert (st == 0).all()
    for A, g, l in zip(mats, G, lp):
        want = np.linalg.inv(A).T / 2
        # reduction, Q and one product of a well-conditioned matrix: a modest multiple of sqrt(n) eps
        assert np.linalg.norm(g - want) <= 32 * np.sqrt(len(A)) * EPS * np.linalg.norm(want), len(A)
        assert np.array_equal(g, -g.T)
        assert abs(l - np.linalg.slogdet(A)[1] / 2) <= 1e-12 * max(1.0, abs(l))


def test_odd_zero_and_small_matrices_in_one_batch():
    mats = [_skew(130, 1, 2.0), _skew(131, 2), np.zeros((140, 140)), _skew(32, 3, 2.0), _skew(257, 4), _skew(200, 5, 2.0)]
    G, lp, sg, st = _run(mats)
    for b in (1, 2, 4):
        assert np.isnan(G[b]).all() and st[b] != 0 and sg[b] == 0
    for b in (0, 3, 5):
        want = np.linalg.inv(mats[b]).T / 2
        assert st[b] == 0 and np.linalg.norm(G[b] - want) <= 1e-12 * np.linalg.norm(want)


def test_replay_with_new_contents():
    import skewgpu

    mats = [_skew(n, 50 + n, 2.0) for n in (150, 220)]
    dA = [skewgpu.to_device(A) for A in mats]
    dG = [torch.zeros_like(a) for a in dA]
    plan = skewgpu.BatchPlan([150, 220])
    pa, pg = plan.pointer_array(dA), plan.pointer_array(dG)
    for seed in (0, 1):
        for a, n in zip(dA, (150, 220)):
            a.copy_(skewgpu.to_device(_skew(n, 1000 * seed + n, 2.0)))
        plan.logabspfaffian(pa, pg)
        for G, n in zip(dG, (150, 220)):
            want = np.linalg.inv(_skew(n, 1000 * seed + n, 2.0)).T / 2
            assert np.linalg.norm(skewgpu.from_device(G) - want) <= 1e-12 * np.linalg.norm(want)
    plan.close()


def test_badly_conditioned_against_oracle():
    """Random matrices (condition up to about 1e5): the error against the binary128 inverse stays
    within the condition number's share, as the host-buffer call's FP64 kernel has it."""
    import skewgpu
    from oracle import oracle as O

    mats = [_skew(128, 600 + k) for k in range(6)]
    G, *_ = _run(mats)
    plan = skewgpu.BatchPlan([128] * 6)
    hA = torch.from_numpy(np.concatenate([A.ravel(order="F") for A in mats])).pin_memory()
    hG = torch.zeros_like(hA).pin_memory()
    plan.logabspfaffian_host(hA, hG)
    plan.close()
    fused = hG.numpy().reshape(6, 128, 128).transpose(0, 2, 1)
    for A, g, f in zip(mats, G, fused):
        want = O.logabspfaffian_grad(A)
        err, ref = np.linalg.norm(g - want) / np.linalg.norm(want), np.linalg.norm(f - want) / np.linalg.norm(want)
        assert err <= 4 * np.linalg.cond(A) * EPS and ref <= 4 * np.linalg.cond(A) * EPS * 4
