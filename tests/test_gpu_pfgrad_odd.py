"""Odd sizes in a gradient batch have no Pfaffian (-inf, sign 0, NaN gradient, singular): they are not
reduced, and the even matrices beside them are as ever."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _batch(skewgpu, sizes):
    gen = torch.Generator(device="cuda").manual_seed(sum(sizes[:8]))
    devs = []
    for n in sizes:
        B = torch.randn(n, n, generator=gen, dtype=torch.float64, device="cuda") / n ** 0.5
        devs.append((B - B.T) / 2)
    grads = [torch.zeros_like(d) for d in devs]
    plan = skewgpu.BatchPlan(sizes)
    out = [torch.zeros(len(sizes), dtype=torch.float64, device="cuda") for _ in range(2)]
    st = torch.zeros(len(sizes), dtype=torch.int32, device="cuda")
    ptrs = plan.pointer_array(devs), plan.pointer_array(grads)

    def call():
        plan.logabspfaffian(*ptrs, *out, st)

    return devs, grads, out, st, call


def test_results(skewgpu):
    sizes = [98, 99, 255, 256, 131, 40, 41]
    devs, grads, (lp, sg), st, call = _batch(skewgpu, sizes)
    call()
    torch.cuda.synchronize()
    for b, n in enumerate(sizes):
        if n % 2:
            assert lp[b] == -np.inf and sg[b] == 0 and st[b] == skewgpu._lib.SKEW_SINGULAR
            assert torch.isnan(grads[b]).all()
        else:
            want = torch.linalg.inv(devs[b]).T / 2
            eps = np.finfo(float).eps
            cond = float(torch.linalg.cond(devs[b]))
            assert st[b] == 0
            assert float(torch.linalg.norm(grads[b] - want)) <= 40 * n * eps * cond * float(torch.linalg.norm(want))


def test_odd_sizes_cost_no_reduction(skewgpu):
    def ms(n):
        call = _batch(skewgpu, [n] * 1024)[-1]
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[1:])

    # a reduction and a gradient of n = 256 each against filling n = 255 with NaN
    assert ms(255) <= ms(256) / 5
