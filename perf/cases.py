"""Performance cases: the calls that a program using this library makes.

Seven kinds of work, each through a public entry point (the Workspace methods,
or the C ABI's device products where the operands are already on the GPU):

  gemm      C := beta C + alpha A B, real or complex, from host arrays or from
            operands on the GPU; square and ragged shapes, 16..2048 a side
  expm      exp(A) of one host matrix, n 8..1024, ||A||_1 from 1e-2 (lowest
            Pade degree) to 1e3 (degree 13 and squarings)
  sweep     exp(A_k) of a frequency sweep A_k = -(G_k + i w_k C_k) on the GPU,
            w up to 1e6, plain FP64 or the split-precision form
  lu        factor, solve (or solve with the adjoint), reciprocal condition
  mixed     the precision form of the solve: low-precision LU and refinement
  expmv     exp(t A_k) B_k of a frequency sweep on the GPU
  gradient  ||exp(tA)B - Y||_F^2 with its gradients in A, B and t

A program keeps one Workspace and puts many matrices through it, so the
Workspace is made once per option and kept.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from csharp_linearalgebra_b200 import Workspace

_WORKSPACES: dict = {}


def _workspace(moduli: int = 0) -> Workspace:
    """The program's workspace; one more for the split-precision form."""
    ws = _WORKSPACES.get(moduli)
    if ws is None:
        ws = _WORKSPACES[moduli] = Workspace()
        if moduli:
            ws.set_split_moduli(moduli)
    return ws


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # One small exponential per call (a time step of a small linear system): latency and launches count.
        dict(name="expm_real_37", kind="expm", cplx=False, n=37, norm=2.0),
        # The dense path at n = 512: one complex exponential of moderate norm.
        dict(name="expm_complex_512", kind="expm", cplx=True, n=512, norm=40.0),
        # The FP64 product at 1024^3 with the operands on the GPU.
        dict(name="gemm_real_1024_device", kind="gemm", cplx=False, device=True, m=1024, n=1024, k=1024,
             alpha=1.0, beta=0.0),
        # A ragged complex product of host arrays, accumulated into C.
        dict(name="gemm_complex_ragged_host", kind="gemm", cplx=True, device=False, m=701, n=513, k=390,
             alpha=-0.5, beta=1.0),
        # A frequency sweep in the reference's own arithmetic: the benchmark's orders, a quarter of its length.
        dict(name="sweep_fp64_64", kind="sweep", count=64, lo=64, hi=1024, wmax=1e6, moduli=0),
        # Half the benchmark's sweep in the split-precision form at its 17 moduli.
        dict(name="sweep_split_128", kind="sweep", count=128, lo=64, hi=1024, wmax=1e6, moduli=17),
        # The dense path at n = 512: factor, solve 8 right-hand sides, condition; real.
        dict(name="lu_real_512", kind="lu", cplx=False, n=512, nrhs=8, adjoint=False, rcond=True),
        # The same for a complex matrix of odd order, solved with the adjoint.
        dict(name="lu_complex_389", kind="lu", cplx=True, n=389, nrhs=3, adjoint=True, rcond=True),
        # A large FP64 factorization with 64 right-hand sides.
        dict(name="lu_real_4096", kind="lu", cplx=False, n=4096, nrhs=64, adjoint=False, rcond=False),
        # The precision form of that solve, moderately conditioned.
        dict(name="mixed_real_4096", kind="mixed", n=4096, nrhs=64, kappa=1e6),
        # The exponential action over a sweep: 8-column panels, the long Taylor recurrences.
        dict(name="expmv_sweep_24", kind="expmv", count=24, lo=64, hi=1024, cols=8, t=0.5, wmax=1e3),
        # The differentiation form: loss and gradients, the backward direction of the exponential action.
        dict(name="gradient_real_600", kind="gradient", cplx=False, n=600, cols=16, norm=60.0),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi], odd ones among them."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "expm", "expm", "sweep", "sweep", "lu", "lu", "mixed", "expmv", "gradient"])
    if kind == "gemm":
        return dict(kind=kind, cplx=rng.random() < 0.5, device=rng.random() < 0.5, m=_log_int(rng, 16, 2048),
                    n=_log_int(rng, 16, 2048), k=_log_int(rng, 16, 2048), alpha=rng.choice([1.0, -0.5]),
                    beta=rng.choice([0.0, 1.0]))
    if kind == "expm":
        return dict(kind=kind, cplx=rng.random() < 0.5, n=_log_int(rng, 8, 1024),
                    norm=round(math.exp(rng.uniform(math.log(1e-2), math.log(1e3))), 4))
    if kind == "sweep":
        lo = _log_int(rng, 16, 128)
        return dict(kind=kind, count=_log_int(rng, 4, 64), lo=lo, hi=_log_int(rng, max(200, lo), 1024),
                    wmax=rng.choice([1e4, 1e6]), moduli=rng.choice([0, 17]))
    if kind == "lu":
        n = _log_int(rng, 24, 3000)
        return dict(kind=kind, cplx=n <= 1400 and rng.random() < 0.5, n=n, nrhs=_log_int(rng, 1, 64),
                    adjoint=rng.random() < 0.5, rcond=n <= 1000)
    if kind == "mixed":
        return dict(kind=kind, n=_log_int(rng, 512, 4096), nrhs=_log_int(rng, 1, 64),
                    kappa=rng.choice([1e2, 1e4, 1e6]))
    if kind == "expmv":
        lo = _log_int(rng, 16, 128)
        return dict(kind=kind, count=_log_int(rng, 2, 24), lo=lo, hi=_log_int(rng, max(200, lo), 1024),
                    cols=_log_int(rng, 1, 16), t=round(rng.uniform(0.1, 0.5), 3), wmax=rng.choice([300.0, 1e3]))
    return dict(kind=kind, cplx=rng.random() < 0.5, n=_log_int(rng, 32, 800), cols=_log_int(rng, 1, 16),
                norm=round(math.exp(rng.uniform(math.log(1.0), math.log(300.0))), 3))


def _sweep_sizes(case):
    """The sweep's orders, evenly over [lo, hi] in a scattered order, and its
    frequencies, log-spaced from 1e2 to wmax."""
    count, lo, hi = case["count"], case["lo"], case["hi"]
    step = next(s for s in range(max(2, int(0.618 * count)), 2 * count + 3) if math.gcd(s, count) == 1)
    orders = [lo + round((hi - lo) * ((i * step) % count) / max(1, count - 1)) for i in range(count)]
    omegas = [10.0 ** (2.0 + (math.log10(case["wmax"]) - 2.0) * i / max(1, count - 1)) for i in range(count)]
    return orders, omegas


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _host(rng, shape, cplx, scale=1.0):
    a = rng.standard_normal(shape)
    if cplx:
        a = (a + 1j * rng.standard_normal(shape)) / math.sqrt(2.0)
    return np.asfortranarray(a * scale)


def _one_norm_matrix(rng, n, cplx, norm):
    """A dense N(0,1) matrix scaled to ||A||_1 = norm."""
    a = _host(rng, (n, n), cplx)
    return np.asfortranarray(a * (norm / np.abs(a).sum(axis=0).max()))


def _sweep_matrices(case, gen):
    """One flat device buffer holding every A_k column-major, and the views.
    A view is the row-major transpose of its matrix; G is as random transposed
    and C is symmetric."""
    orders, omegas = _sweep_sizes(case)
    flat = torch.empty(sum(n * n for n in orders), dtype=torch.complex128, device="cuda")
    views, at = [], 0
    for n, w in zip(orders, omegas):
        v = flat[at:at + n * n].view(n, n)
        g = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen) / math.sqrt(n)
        q, _ = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen))
        d = torch.exp(torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * -math.log(1e-3)
                      + math.log(1e-3))
        c = (q.T * d) @ q
        c = 0.5 * (c + c.T)
        v.copy_(torch.complex(-g, -w * c))
        views.append(v)
        at += n * n
    return orders, flat, views


def _conditioned(case, gen):
    """A = U diag(sigma) V^T with sigma log-spaced from 1 to 1/kappa, on the GPU."""
    n = case["n"]
    u, _ = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen))
    v, _ = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen))
    s = torch.logspace(0.0, -math.log10(case["kappa"]), n, dtype=torch.float64, device="cuda")
    return (u * s) @ v.T


def _inputs(case, seed):
    """The inputs alone, without a workspace (exact() starts from them too)."""
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "gemm":
        m, n, k, cplx = case["m"], case["n"], case["k"], case["cplx"]
        if case["device"]:
            dt = torch.complex128 if cplx else torch.float64
            # row-major transposes: the column-major operands
            return dict(a=torch.randn(k, m, dtype=dt, device="cuda", generator=gen),
                        b=torch.randn(n, k, dtype=dt, device="cuda", generator=gen),
                        c=torch.randn(n, m, dtype=dt, device="cuda", generator=gen))
        return dict(a=_host(rng, (m, k), cplx), b=_host(rng, (k, n), cplx), c=_host(rng, (m, n), cplx))
    if kind == "expm":
        return dict(a=_one_norm_matrix(rng, case["n"], case["cplx"], case["norm"]))
    if kind == "sweep":
        orders, flat, views = _sweep_matrices(case, gen)
        return dict(orders=orders, flat=flat, views=views)
    if kind == "lu":
        n = case["n"]
        return dict(a=_host(rng, (n, n), case["cplx"], 1.0 / math.sqrt(n)),
                    b=_host(rng, (n, case["nrhs"]), case["cplx"]))
    if kind == "mixed":
        a = _conditioned(case, gen)
        return dict(a=np.asfortranarray(a.cpu().numpy()), b=_host(rng, (case["n"], case["nrhs"]), False))
    if kind == "expmv":
        orders, flat, views = _sweep_matrices(case, gen)
        c = case["cols"]
        b = torch.randn(sum(orders) * c, dtype=torch.complex128, device="cuda", generator=gen)
        return dict(orders=orders, flat=flat, views=views, b=b)
    n, c, cplx = case["n"], case["cols"], case["cplx"]
    return dict(a=_one_norm_matrix(rng, n, cplx, case["norm"]), b=_host(rng, (n, c), cplx),
                y=_host(rng, (n, c), cplx))


def _panels(flat, orders, cols):
    """The column-major n_k x cols panels of a flat buffer, as row-major cols x n_k views."""
    views, at = [], 0
    for n in orders:
        views.append(flat[at:at + n * cols].view(cols, n))
        at += n * cols
    return views


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"] = case
    state["ws"] = _workspace(case.get("moduli", 0))
    kind = case["kind"]
    if kind == "gemm" and case["device"]:
        # alpha and beta of a complex product are (re, im) pairs in memory
        state["alpha"] = np.array([case["alpha"], 0.0])
        state["beta"] = np.array([case["beta"], 0.0])
        state["out"] = torch.empty_like(state["c"])
    if kind == "sweep":
        state["out"] = torch.empty_like(state["flat"])
        o, at = [], 0
        for n in state["orders"]:
            o.append(state["out"][at:at + n * n].data_ptr())
            at += n * n
        state["a_ptrs"], state["o_ptrs"] = [v.data_ptr() for v in state["views"]], o
    if kind == "expmv":
        state["out"] = torch.empty_like(state["b"])
        state["a_ptrs"] = [v.data_ptr() for v in state["views"]]
        state["b_ptrs"] = [v.data_ptr() for v in _panels(state["b"], state["orders"], case["cols"])]
        state["o_ptrs"] = [v.data_ptr() for v in _panels(state["out"], state["orders"], case["cols"])]
    if kind in ("gemm", "sweep", "expmv"):
        # The library works on its own stream: the inputs are complete before its calls.
        torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(state):
    case, ws = state["case"], state["ws"]
    kind = case["kind"]
    if kind == "gemm":
        if not case["device"]:
            return ws.multiply(state["a"], state["b"], state["c"], case["alpha"], case["beta"])
        m, n, k = case["m"], case["n"], case["k"]
        a, b, out = state["a"], state["b"], state["out"]
        if case["beta"] != 0.0:
            # The accumulated product overwrites its C: each pass starts from the same one.
            out.copy_(state["c"])
            torch.cuda.current_stream().synchronize()
        if case["cplx"]:
            ws._call("tns_zgemm_device", m, n, k, state["alpha"].ctypes.data_as(ctypes.c_void_p), a.data_ptr(), m,
                     b.data_ptr(), k, state["beta"].ctypes.data_as(ctypes.c_void_p), out.data_ptr(), m)
        else:
            ws._call("tns_dgemm_device", m, n, k, case["alpha"], a.data_ptr(), m, b.data_ptr(), k, case["beta"],
                     out.data_ptr(), m)
        return out
    if kind == "expm":
        return ws.expm(state["a"])
    if kind == "sweep":
        orders = state["orders"]
        info = ws.expm_batched_device(len(orders), orders, state["a_ptrs"], orders, state["o_ptrs"], orders)
        return {"exp": state["out"], "degrees": np.array([(i.degree, i.squarings) for i in info])}
    if kind == "lu":
        lu = ws.factor_lu(state["a"])
        x = lu.solve_adjoint(state["b"]) if case["adjoint"] else lu.solve(state["b"])
        out = {"factors": lu.factors, "pivots": lu.pivots, "x": x}
        if case["rcond"]:
            out["rcond"] = lu.reciprocal_condition()
        return out
    if kind == "mixed":
        x, _ = ws.solve_mixed(state["a"], state["b"])
        return x
    if kind == "expmv":
        orders = state["orders"]
        info = ws.expmv_batched_device(len(orders), orders, state["a_ptrs"], orders, case["cols"], state["b_ptrs"],
                                       orders, case["t"], state["o_ptrs"], orders)
        return {"f": state["out"], "counts": np.array([(i.degree, i.scaling, i.applications) for i in info])}
    g = ws.expmv_gradient(state["a"], state["b"], state["y"])
    return {"loss": g["loss"], "f": g["f"], "grad_a": g["grad_a"], "grad_b": g["grad_b"], "grad_t": g["grad_t"]}


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------

def _expm_flops(n, norm, cplx):
    """Degree 13 with s squarings, or a lower degree of fewer products, and the Pade solve."""
    s = max(0, math.ceil(math.log2(norm / 4.25))) if norm > 0 else 0
    products = 6 + s if norm >= 2.1 else 5 if norm >= 0.95 else 4 if norm >= 0.25 else 3 if norm >= 0.015 else 2
    return (4.0 if cplx else 1.0) * (2.0 * products + 8.0 / 3.0) * float(n) ** 3


def work(case):
    kind = case["kind"]
    z = 16.0 if case.get("cplx") else 8.0
    mul = 4.0 if case.get("cplx") else 1.0
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": z * (m * k + k * n + m * n * (1 + (case["beta"] != 0.0))), "flops": mul * 2.0 * m * n * k}
    if kind == "expm":
        n = case["n"]
        # A dense random matrix: ||A^p||^(1/p) is near its spectral radius, about ||A||_1 / sqrt(0.64 n).
        return {"bytes": z * 2 * n * n, "flops": _expm_flops(n, case["norm"] * 1.25 / math.sqrt(n), case["cplx"])}
    if kind == "sweep":
        orders, omegas = _sweep_sizes(case)
        return {"bytes": 32.0 * sum(n * n for n in orders),
                "flops": sum(_expm_flops(n, w, True) for n, w in zip(orders, omegas))}
    if kind == "lu":
        n, r = case["n"], case["nrhs"]
        return {"bytes": z * (2 * n * n + 2 * n * r),
                "flops": mul * (2.0 / 3.0 * n ** 3 + 2.0 * n * n * (r + (16 if case["rcond"] else 0)))}
    if kind == "mixed":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8.0 * (n * n + 2 * n * r), "flops": 2.0 / 3.0 * n ** 3 + 4.0 * n * n * r}
    if kind == "expmv":
        orders, omegas = _sweep_sizes(case)
        c = case["cols"]
        # about 1.2 |t| ||A|| applications, and never fewer than a dozen
        apps = [max(12.0, 1.2 * case["t"] * w) for w in omegas]
        return {"bytes": 16.0 * sum(n * n + 2 * n * c for n in orders),
                "flops": sum(8.0 * n * n * c * a for n, a in zip(orders, apps))}
    n, c = case["n"], case["cols"]
    return {"bytes": z * (2 * n * n + 4 * n * c), "flops": 3.0 * _expm_flops(n, case["norm"], case["cplx"])}


# ---------------------------------------------------------------------------
# The same results from plain torch and numpy in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "gemm":
        if case["device"]:
            r = case["alpha"] * (x["b"] @ x["a"])
            return r + case["beta"] * x["c"] if case["beta"] != 0.0 else r
        return np.asfortranarray(case["alpha"] * (x["a"] @ x["b"]) + case["beta"] * x["c"])
    if kind == "expm":
        return torch.linalg.matrix_exp(torch.from_numpy(np.ascontiguousarray(x["a"])).cuda()).cpu().numpy()
    if kind == "sweep":
        return {"exp": torch.cat([torch.linalg.matrix_exp(v).reshape(-1) for v in x["views"]]), "degrees": None}
    if kind == "lu":
        a = torch.from_numpy(np.ascontiguousarray(x["a"])).cuda()
        a = a.mH if case["adjoint"] else a
        b = torch.from_numpy(np.ascontiguousarray(x["b"])).cuda()
        out = {"factors": None, "pivots": None, "x": torch.linalg.solve(a, b).cpu().numpy()}
        if case["rcond"]:
            out["rcond"] = None  # an estimate
        return out
    if kind == "mixed":
        a = torch.from_numpy(np.ascontiguousarray(x["a"])).cuda()
        b = torch.from_numpy(np.ascontiguousarray(x["b"])).cuda()
        y = torch.linalg.solve(a, b)
        return (y + torch.linalg.solve(a, b - a @ y)).cpu().numpy()
    if kind == "expmv":
        # the views are transposes: F^T = B^T exp(t A)^T
        bs = _panels(x["b"], x["orders"], case["cols"])
        return {"f": torch.cat([(b @ torch.linalg.matrix_exp(case["t"] * v)).reshape(-1)
                                for b, v in zip(bs, x["views"])]), "counts": None}
    a, b, y = (torch.from_numpy(np.ascontiguousarray(x[q])).cuda() for q in ("a", "b", "y"))
    a, b = a.requires_grad_(), b.requires_grad_()
    t = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    f = torch.linalg.matrix_exp(t * a) @ b
    loss = (f - y).abs().square().sum()
    ga, gb, gt = torch.autograd.grad(loss, (a, b, t))
    return {"loss": float(loss), "f": f.detach().cpu().numpy(), "grad_a": ga.cpu().numpy(),
            "grad_b": gb.cpu().numpy(), "grad_t": float(gt)}
