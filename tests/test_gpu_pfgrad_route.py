"""Whether a batch's gradients are formed on the tensor cores depends on its size and, from a matrix per
SM on, on how its sizes fill the tiles."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("sizes", [[98, 106, 99], [98, 108], [128, 130], [130, 136, 131], [130, 138], [138],
                                   [98, 107, 108, 128, 130, 142, 148, 200, 131, 256, 40]])
@pytest.mark.parametrize("copies", [1, 150])
def test_both_forms(skewgpu, sizes, copies):
    gen = torch.Generator(device="cuda").manual_seed(1)
    one = []
    for n in sizes:
        B = torch.randn(n, n, generator=gen, dtype=torch.float64, device="cuda") / n ** 0.5
        A = (B - B.T) / 2
        k = torch.arange(0, n - 1, 2, device="cuda")
        A[k, k + 1] += 2.0
        A[k + 1, k] -= 2.0
        one.append(A)
    devs = one * copies
    grads = [torch.full_like(d, 7.0) for d in devs]
    plan = skewgpu.BatchPlan(sizes * copies)
    for _ in range(2):
        lp, sg, st = plan.logabspfaffian(plan.pointer_array(devs), plan.pointer_array(grads))
    torch.cuda.synchronize()
    lp = lp.cpu().numpy()
    for b, n in enumerate(sizes * copies):
        G, A = grads[b], devs[b]
        if n % 2:
            assert torch.isnan(G).all() and lp[b] == -np.inf
            continue
        want = torch.linalg.inv(A).T / 2
        # reduction, Q and products of a well-conditioned matrix: a modest multiple of sqrt(n) eps
        assert float(torch.linalg.norm(G - want)) <= 32 * np.sqrt(n) * EPS * float(torch.linalg.norm(want)), n
        assert torch.equal(G, -G.T) and lp[b] == lp[b % len(sizes)]
    plan.close()
