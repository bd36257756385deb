"""The workloads whose speed this framework is kept to, over the ranges its users run.

listed() gives the fixed cases, draw(rng) one more case of the same ranges.  A case is
prepared once (prepare: the inputs on the GPU, the plan and the buffers a program keeps),
run any number of times (run: one pass through the public entry points), and checked
against plain torch in 64 bits (exact), which uses none of this package.

Matrices are column-major on the device: a torch tensor T holds A when T[j, i] = A[i, j].
Entries follow the package's own workloads: A = (B - B^T)/2 with B iid normal, with
variance 1/n in the batched Pfaffian and eigenvalue work (the Pfaffian gradients add a
multiple of the symplectic form J, which keeps the matrices well-conditioned), scaled to a
spectral radius of 0.5 to 8 where exp is taken.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "skewlinearalgebra.jl_gb300"))

import skewgpu  # noqa: E402
from skewgpu import _lib  # noqa: E402


def listed():
    return [
        # The smallest call: log|Pf| and sign of one small matrix, answered on the host.
        {"name": "pfaffian_one_16", "do": "pf_one", "n": 16},
        # Many Pfaffians with their gradients, uneven even sizes: the batched solver's main load.
        {"name": "pf_grad_4096_mixed", "do": "pf_grad", "count": 4096, "lo": 16, "hi": 256, "step": 2, "pick": 1},
        # Spectra of the same kind of batch, values only, in the QR's deflation order.
        {"name": "eigvals_4096_mixed", "do": "eigvals_batch", "count": 4096, "lo": 16, "hi": 256, "step": 2,
         "pick": 2},
        # Eigenpairs of a batch of small and middle sizes, odd ones among them.
        {"name": "eigen_256_mixed", "do": "eigen_batch", "count": 256, "lo": 15, "hi": 200, "step": 1, "pick": 3},
        # Training through exp: the adjoint for a batch of sizes 32 .. 512.
        {"name": "exp_vjp_512_mixed", "do": "exp_vjp", "count": 512, "lo": 32, "hi": 512, "step": 32, "pick": 4},
        # The same for complex matrices of one size.
        {"name": "exp_vjp_z_64x256", "do": "exp_vjp_z", "count": 64, "n": 256},
        # Complex skew-symmetric Pfaffians, one size.
        {"name": "pfaffian_z_2048x128", "do": "pf_z", "count": 2048, "n": 128},
        # One middle-sized matrix: the tridiagonalisation alone.
        {"name": "hessenberg_512", "do": "hessenberg", "n": 512},
        # One middle-sized matrix: its spectrum in the QR's deflation order.
        {"name": "eigvals_512", "do": "eigvals", "n": 512},
        # One large matrix: the blocked tridiagonalisation.
        {"name": "hessenberg_8192", "do": "hessenberg", "n": 8192},
        # exp of one large real matrix (eigenpairs, back-transformation, products).
        {"name": "exp_2048", "do": "exp", "n": 2048},
        # exp of one large complex matrix of a ragged size.
        {"name": "exp_z_1501", "do": "exp_z", "n": 1501},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    do = rng.choice(["pf_one", "pf_grad", "eigvals_batch", "eigen_batch", "exp_vjp", "exp_vjp_z", "pf_z",
                     "hessenberg", "eigvals", "exp", "exp_z"])
    pick = rng.randrange(1 << 20)
    if do == "pf_one":
        return {"do": do, "n": 2 * _log_uniform(rng, 2, 128)}
    if do == "pf_grad":
        # uneven batches, and (lo == hi) batches of one size
        lo = 2 * _log_uniform(rng, 4, 64)
        hi = rng.choice([lo, 2 * rng.randint(lo // 2, 128)])
        return {"do": do, "count": _log_uniform(rng, 32, 4096), "lo": lo, "hi": hi, "step": 2, "pick": pick}
    if do == "eigvals_batch":
        lo = rng.randint(8, 64)
        return {"do": do, "count": _log_uniform(rng, 32, 4096), "lo": lo, "hi": rng.randint(lo, 256), "step": 1,
                "pick": pick}
    if do == "eigen_batch":
        lo = rng.randint(8, 64)
        return {"do": do, "count": _log_uniform(rng, 16, 512), "lo": lo, "hi": rng.randint(lo, 256), "step": 1,
                "pick": pick}
    if do == "exp_vjp":
        lo = rng.randint(8, 200)
        return {"do": do, "count": _log_uniform(rng, 8, 512), "lo": lo, "hi": rng.randint(lo, 512), "step": 1,
                "pick": pick}
    if do == "exp_vjp_z":
        return {"do": do, "count": _log_uniform(rng, 4, 64), "n": _log_uniform(rng, 24, 256)}
    if do == "pf_z":
        return {"do": do, "count": _log_uniform(rng, 64, 2048), "n": 2 * _log_uniform(rng, 8, 64)}
    if do == "hessenberg":
        return {"do": do, "n": _log_uniform(rng, 64, 8192)}
    if do == "eigvals":
        return {"do": do, "n": _log_uniform(rng, 32, 700)}
    if do == "exp":
        return {"do": do, "n": _log_uniform(rng, 64, 3000)}
    return {"do": do, "n": _log_uniform(rng, 64, 2048)}


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
def _sizes(case):
    """The batch's sizes: part of the case, not of the seed (a plan fixes them)."""
    rng = np.random.default_rng(case["pick"])
    steps = (case["hi"] - case["lo"]) // case["step"]
    return (case["lo"] + case["step"] * rng.integers(0, steps + 1, case["count"])).astype(np.int64)


def _layout(sizes):
    """(offsets, total, groups): the matrices lie in one buffer, equal sizes next to each other."""
    order = np.argsort(sizes, kind="stable")
    offs = np.zeros(len(sizes), dtype=np.int64)
    offs[order[1:]] = np.cumsum(sizes[order[:-1]] ** 2)
    total = int((sizes ** 2).sum())
    groups = []
    for n in np.unique(sizes):
        members = np.nonzero(sizes == n)[0]
        members = members[np.argsort(offs[members])]
        groups.append((int(n), members, int(offs[members[0]])))
    return offs, total, groups


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed % (1 << 62))


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, dtype=torch.float64, device="cuda")


def _skew_batch(case, seed):
    """The packed batch, and the factor that makes the spectral radius what the path meets."""
    sizes = _sizes(case)
    offs, total, groups = _layout(sizes)
    gen = _gen(seed)
    buf = _randn(gen, total)
    for n, members, at in groups:
        B = buf[at: at + len(members) * n * n].view(len(members), n, n)
        A = (B - B.transpose(1, 2)) / 2
        if case["do"] == "exp_vjp":  # spectral radius about 0.5 .. 8
            r = 0.5 + 7.5 * torch.rand(len(members), 1, 1, generator=gen, dtype=torch.float64, device="cuda")
            A = A * (r / math.sqrt(2.0 * n))
        else:  # variance 1/n before the skew part is taken
            A = A / math.sqrt(n)
            if case["do"] == "pf_grad":  # a pairing term 2 J, which keeps a gradient's matrices well-conditioned
                k = torch.arange(0, n, 2, device="cuda")
                A[:, k, k + 1] -= 2.0
                A[:, k + 1, k] += 2.0
        B.copy_(A)
    return sizes, offs, total, groups, buf, gen


def _skew(n, seed, radius=None):
    gen = _gen(seed)
    B = _randn(gen, n, n)
    A = (B - B.T) / 2
    if radius is not None:
        A = A * (radius / math.sqrt(2.0 * n))
    return A.contiguous()


def _skew_hermitian(count, n, seed):
    """count complex skew-Hermitian matrices with a spectral radius of about 0.5 .. 8."""
    gen = _gen(seed)
    C = torch.complex(_randn(gen, count, n, n), _randn(gen, count, n, n))
    A = (C - C.mH) / 2
    r = 0.5 + 7.5 * torch.rand(count, 1, 1, generator=gen, dtype=torch.float64, device="cuda")
    return (A * (r / (2.0 * math.sqrt(n)))).contiguous(), gen


def _pointers(buf, offs, item=8):
    base = buf.data_ptr()
    return torch.tensor((base + item * offs).tolist(), dtype=torch.int64, device="cuda")


def _vector_offsets(sizes):
    offs = np.zeros(len(sizes), dtype=np.int64)
    offs[1:] = np.cumsum(sizes[:-1])
    return offs


def prepare(case, seed):
    do = case["do"]
    if do in ("pf_grad", "eigvals_batch", "eigen_batch", "exp_vjp"):
        sizes, offs, total, groups, buf, gen = _skew_batch(case, seed)
        s = {"do": do, "buf": buf, "A": _pointers(buf, offs), "plan": skewgpu.BatchPlan(sizes),
             "status": torch.zeros(len(sizes), dtype=torch.int32, device="cuda")}
        vals = torch.zeros(int(sizes.sum()), dtype=torch.float64, device="cuda")
        if do == "pf_grad":
            s["grad"] = torch.zeros_like(buf)
            s["G"] = _pointers(s["grad"], offs)
            s["logpf"] = torch.zeros(len(sizes), dtype=torch.float64, device="cuda")
            s["sign"] = torch.zeros_like(s["logpf"])
        elif do == "eigvals_batch":
            s["vals"], s["V"] = vals, _pointers(vals, _vector_offsets(sizes))
        elif do == "eigen_batch":
            s["vals"], s["V"] = vals, _pointers(vals, _vector_offsets(sizes))
            s["re"], s["im"] = torch.zeros_like(buf), torch.zeros_like(buf)
            s["Vr"], s["Vi"] = _pointers(s["re"], offs), _pointers(s["im"], offs)
        else:
            s["cot"] = _randn(gen, total)
            s["grad"] = torch.zeros_like(buf)
            s["C"], s["G"] = _pointers(s["cot"], offs), _pointers(s["grad"], offs)
        return s
    n = case["n"]
    if do in ("pf_one", "hessenberg"):
        return {"do": do, "A": skewgpu.SkewHermitian(_skew(n, seed))}
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    if do == "eigvals":
        return {"do": do, "n": n, "A": _skew(n, seed), "info": info,
                "vals": torch.zeros(n, dtype=torch.float64, device="cuda")}
    if do == "exp":
        A = _skew(n, seed, radius=4.0)
        return {"do": do, "n": n, "A": A, "E": torch.zeros_like(A), "info": info}
    if do == "exp_z":
        A = _skew_hermitian(1, n, seed)[0][0].contiguous()
        return {"do": do, "n": n, "A": A, "E": torch.zeros_like(A), "info": info}
    count = case["count"]
    if do == "exp_vjp_z":
        A, gen = _skew_hermitian(count, n, seed)
        C = torch.complex(_randn(gen, count, n, n), _randn(gen, count, n, n))
        return {"do": do, "n": n, "count": count, "A": A, "C": C, "G": torch.zeros_like(A)}
    gen = _gen(seed)  # pf_z: A == -transpose(A)
    C = torch.complex(_randn(gen, count, n, n), _randn(gen, count, n, n))
    return {"do": do, "A": ((C - C.mT) / 2).contiguous(),
            "logpf": torch.zeros(count, dtype=torch.float64, device="cuda"),
            "phase": torch.zeros(count, dtype=torch.complex128, device="cuda"),
            "status": torch.zeros(count, dtype=torch.int32, device="cuda"), "n": n, "count": count}


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _c_abi():
    """The library's C interface and the current device's handle on the current stream."""
    return _lib.load(), skewgpu.handle().bind()


def run(s):
    do = s["do"]
    if do == "pf_one":
        lp, sg = skewgpu.logabspfaffian(s["A"])
        return {"logpf": lp, "sign": sg}
    if do == "hessenberg":
        F = skewgpu.hessenberg(s["A"])
        # the reflectors' entries below their leading one
        return {"reflectors": torch.triu(F.factors, 2), "tau": F.tau, "ev": F.ev}
    if do == "pf_grad":
        s["plan"].logabspfaffian(s["A"], s["G"], s["logpf"], s["sign"], s["status"])
        return {"logpf": s["logpf"], "sign": s["sign"], "grad": s["grad"], "status": s["status"]}
    if do == "eigvals_batch":
        s["plan"].eigvals(s["A"], s["V"], s["status"])
        return {"vals": s["vals"], "status": s["status"]}
    if do == "eigen_batch":
        s["plan"].eigen(s["A"], s["V"], s["Vr"], s["Vi"], s["status"])
        return {"vals": s["vals"], "re": s["re"], "im": s["im"], "status": s["status"]}
    if do == "exp_vjp":
        s["plan"].exp_vjp(s["A"], s["C"], s["G"], s["status"])
        return {"grad": s["grad"], "status": s["status"]}
    lib, h = _c_abi()
    n = s["n"]
    if do == "exp_vjp_z":
        _lib.check(lib.skew_batch_exp_vjp_z(h, _p(s["A"]), n, s["count"], _p(s["C"]), _p(s["G"]), None))
        return {"grad": s["G"]}
    if do == "pf_z":
        _lib.check(lib.skew_batch_logabspf_z(h, _p(s["A"]), n, s["count"], _p(s["logpf"]), _p(s["phase"]), None, 1,
                                             _p(s["status"])))
        return {"logpf": s["logpf"], "phase": s["phase"], "status": s["status"]}
    work = s["A"].clone()  # the single-matrix calls work in place
    if do == "eigvals":
        _lib.check(lib.skew_eigvals_d(h, _p(work), n, n, _p(s["vals"]), _p(s["info"])))
        return {"vals": s["vals"], "info": s["info"]}
    call = lib.skew_exp_d if do == "exp" else lib.skew_exp_z
    _lib.check(call(h, _p(work), n, n, _p(s["E"]), n, _p(s["info"])))
    return {"exp": s["E"]}


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    do = case["do"]
    if "pick" in case:
        n = _sizes(case).astype(np.float64)
    else:
        n = np.full(case.get("count", 1), case["n"], dtype=np.float64)
    n2, n3, n1 = float((n ** 2).sum()), float((n ** 3).sum()), float(n.sum())
    reduce, count = 4.0 / 3.0 * n3, len(n)
    if do == "pf_one":
        return {"bytes": 8 * n2 + 16 * count, "flops": reduce}
    if do == "pf_grad":
        return {"bytes": 16 * n2 + 20 * count, "flops": reduce + 2 * n3}
    if do in ("eigvals_batch", "eigvals"):
        return {"bytes": 8 * n2 + 8 * n1 + 4 * count, "flops": reduce}
    if do == "eigen_batch":
        return {"bytes": 24 * n2 + 8 * n1 + 4 * count, "flops": reduce + 4.0 / 3.0 * n3 + 4 * n3}
    if do == "exp_vjp":
        return {"bytes": 24 * n2 + 4 * count, "flops": reduce + 2 * n3 + 8 * n3}
    if do == "exp_vjp_z":
        return {"bytes": 48 * n2, "flops": 4 * (reduce + 2 * n3 + 8 * n3)}
    if do == "pf_z":
        return {"bytes": 16 * n2 + 28 * count, "flops": reduce}
    if do == "hessenberg":
        return {"bytes": 8 * n2 + 4 * n2 + 16 * n1, "flops": reduce}
    if do == "exp":
        return {"bytes": 16 * n2, "flops": reduce + 2 * n3 + 2 * n3}
    return {"bytes": 32 * n2, "flops": 4 * (reduce + 2 * n3 + 2 * n3)}


# ---------------------------------------------------------------------------------------
# The same in 64 bits by plain torch
# ---------------------------------------------------------------------------------------
def _hessenberg_64(T):
    """Householder tridiagonalisation of a real skew matrix, one column at a time."""
    A = T.clone().T.contiguous()  # row-major A
    n = A.shape[0]
    R = torch.zeros_like(A)
    tau = torch.zeros(max(n - 1, 0), dtype=torch.float64, device="cuda")
    ev = torch.zeros_like(tau)
    for k in range(n - 1):
        x = A[k + 1:, k].clone()
        if n - 1 - k == 1:
            ev[k] = x[0]
            R[k + 1, k] = 1.0
            continue
        alpha, rest = x[0], torch.linalg.vector_norm(x[1:])
        beta = -torch.copysign(torch.hypot(alpha, rest), alpha)
        t = 1.0 - alpha / beta
        v = x / (alpha - beta)
        v[0] = 1.0
        W = A[k + 1:, k + 1:]
        p = t * (W @ v)
        W.addr_(p, v, alpha=-1.0)
        W.addr_(v, p)
        R[k + 1:, k] = v  # with its leading one
        tau[k] = t
        ev[k] = beta
    return R.T.contiguous(), tau, ev


def _frechet_64(A, C):
    """sum of exp's adjoint: the upper right block of exp([[A^H, C], [0, A^H]]), batched."""
    n = A.shape[-1]
    M = torch.zeros(*A.shape[:-2], 2 * n, 2 * n, dtype=A.dtype, device=A.device)
    M[..., :n, :n] = A.mH
    M[..., n:, n:] = A.mH
    M[..., :n, n:] = C
    return torch.matrix_exp(M)[..., :n, n:]


def exact(case, seed):
    do = case["do"]
    if do == "pf_one":
        A = _skew(case["n"], seed)
        return {"logpf": float(torch.linalg.slogdet(A)[1]) / 2, "sign": None}
    if do == "hessenberg":
        R, tau, ev = _hessenberg_64(_skew(case["n"], seed))
        return {"reflectors": torch.triu(R, 2), "tau": tau, "ev": ev}
    if do == "pf_grad":
        sizes, offs, total, groups, buf, _ = _skew_batch(case, seed)
        logpf = torch.zeros(len(sizes), dtype=torch.float64, device="cuda")
        grad = torch.zeros_like(buf)
        for n, members, at in groups:
            T = buf[at: at + len(members) * n * n].view(len(members), n, n)
            logpf[torch.from_numpy(members).cuda()] = torch.linalg.slogdet(T)[1] / 2
            # T = A^T, and the gradient 1/2 A^{-T} is stored transposed too: 1/2 A^{-1} = 1/2 inv(T)^T
            grad[at: at + len(members) * n * n] = (torch.linalg.inv(T) / 2).mT.reshape(-1)
        return {"logpf": logpf, "sign": None, "grad": grad, "status": None}
    if do == "exp_vjp":
        sizes, offs, total, groups, buf, gen = _skew_batch(case, seed)
        cot = _randn(gen, total)
        grad = torch.zeros_like(buf)
        for n, members, at in groups:
            for b in range(0, len(members), 64):
                lo, hi = at + b * n * n, at + min(b + 64, len(members)) * n * n
                A = buf[lo:hi].view(-1, n, n).mT
                C = cot[lo:hi].view(-1, n, n).mT
                grad[lo:hi] = _frechet_64(A, C).mT.reshape(-1)
        return {"grad": grad, "status": None}
    if do == "exp_vjp_z":
        A, gen = _skew_hermitian(case["count"], case["n"], seed)
        n, count = case["n"], case["count"]
        C = torch.complex(_randn(gen, count, n, n), _randn(gen, count, n, n))
        G = [_frechet_64(A[b: b + 16].mT, C[b: b + 16].mT).mT for b in range(0, count, 16)]
        return {"grad": torch.cat(G).contiguous()}
    if do == "pf_z":
        gen = _gen(seed)
        n, count = case["n"], case["count"]
        C = torch.complex(_randn(gen, count, n, n), _randn(gen, count, n, n))
        return {"logpf": torch.linalg.slogdet((C - C.mT) / 2)[1] / 2, "phase": None, "status": None}
    if do == "exp":
        return {"exp": torch.matrix_exp(_skew(case["n"], seed, radius=4.0))}
    if do == "exp_z":
        return {"exp": torch.matrix_exp(_skew_hermitian(1, case["n"], seed)[0][0])}
    return None  # eigenvalues in deflation order and eigenvectors' phases are the algorithm's own
