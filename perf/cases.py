"""The engine's work as its users call it, for timing: cases, their inputs,
one pass through the public entry points, the work of a pass, and the same
results in plain 64-bit torch.

    listed()             the cases that are always timed
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs (on the GPU, or on the host where the entry takes host arrays)
    run(state)           one pass, returning its outputs
    work(case)           bytes and operations that a pass cannot do without
    exact(case, seed)    the outputs of run() from plain float64 torch

The stopping error is not among the outputs: it is a difference of nearly equal
numbers, whose digits say nothing once a solve has converged; the iteration
count, which follows from it, is there.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import rwig_b200 as rw
from rwig_b200 import _lib

DEV = "cuda"
F64 = torch.float64


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small vanilla solve on resident data: launch and barrier latency
        {"name": "vanilla_256", "kind": "vanilla", "m": 256, "n": 256, "d": 2, "alpha": 1.0, "reg": 0.1,
         "max_iter": 1000, "tol": 1e-9, "plan": True, "grad": False},
        # the R-facing call on host arrays, odd sizes, method chosen by the "auto" rule
        {"name": "host_120x95", "kind": "host", "m": 120, "n": 95, "d": 2, "alpha": 1.0, "reg": 0.1,
         "max_iter": 1000, "tol": 1e-6},
        # an ordinary solve with its plan, odd sizes
        {"name": "log_1777x1501", "kind": "log", "m": 1777, "n": 1501, "d": 3, "alpha": 1.0, "reg": 0.05,
         "max_iter": 2000, "tol": 1e-9, "plan": True, "grad": False},
        # a large solve whose cost matrix exceeds the L2 cache, potentials and loss only
        {"name": "log_4096", "kind": "log", "m": 4096, "n": 4096, "d": 2, "alpha": 0.5, "reg": 0.01,
         "max_iter": 2000, "tol": 1e-9, "plan": False, "grad": False},
        # forward and backward: the gradient of the loss with respect to a, fixed unrolling
        {"name": "log_grad_2048", "kind": "log", "m": 2048, "n": 2048, "d": 2, "alpha": 0.5, "reg": 0.05,
         "max_iter": 100, "tol": 0.0, "plan": False, "grad": True},
        # the same in the vanilla form, small and odd, run to its tolerance
        {"name": "vanilla_grad_701x513", "kind": "vanilla", "m": 701, "n": 513, "d": 3, "alpha": 1.0, "reg": 0.1,
         "max_iter": 200, "tol": 1e-9, "plan": True, "grad": True},
        # log barycenter of 32 histograms with its gradient, fixed unrolling
        {"name": "bary_log_grad_2048x32", "kind": "bary", "log": True, "m": 2048, "n": 2048, "s": 32, "d": 50,
         "reg": 0.05, "max_iter": 50, "tol": 0.0, "grad": True},
        # a small parallel barycenter run to its tolerance, sources and targets of different sizes
        {"name": "bary_par_600x501x7", "kind": "bary", "log": False, "m": 600, "n": 501, "s": 7, "d": 2,
         "reg": 0.1, "max_iter": 500, "tol": 1e-6, "grad": False},
        # a sharp log barycenter: exp(-C/reg) underflows, so every sweep is a soft-min
        {"name": "bary_sharp_grad_360x5", "kind": "bary", "log": True, "m": 360, "n": 360, "s": 5, "d": 2,
         "reg": 0.001, "max_iter": 20, "tol": 0.0, "grad": True},
        # one dictionary-learning gradient: 64 documents over 5000 words, 16 topics
        {"name": "wdl_grad_5000", "kind": "wdl", "n": 5000, "s": 16, "docs": 64, "d": 64, "reg": 0.05, "max_iter": 20},
        # a whole dictionary-learning call on a small corpus: training and inference, host arrays
        {"name": "wdl_train_700", "kind": "train", "n": 700, "s": 6, "docs": 96, "batch": 32, "d": 64, "reg": 0.05,
         "max_iter": 20},
        # 200 solves of mixed sizes in one batched call
        {"name": "stream_200", "kind": "stream", "count": 200, "lo": 64, "hi": 8192, "max_iter": 2000, "tol": 1e-9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vanilla", "host", "log", "log", "grad", "bary", "bary", "sharp", "wdl", "wdl", "train", "stream"])
    if kind == "host":
        return {"kind": "host", "m": _log_int(rng, 40, 600), "n": _log_int(rng, 40, 600), "d": rng.choice([2, 3, 64]),
                "alpha": 1.0, "reg": rng.choice([0.05, 0.1, 0.5]), "max_iter": 1000, "tol": 1e-6}
    if kind in ("vanilla", "log"):
        lo, hi = (64, 2048) if kind == "vanilla" else (64, 6000)
        return {"kind": kind, "m": _log_int(rng, lo, hi), "n": _log_int(rng, lo, hi), "d": rng.choice([2, 3, 64]),
                "alpha": rng.choice([0.5, 1.0]), "reg": rng.choice([0.05, 0.1] if kind == "vanilla" else [0.01, 0.05, 0.1]),
                "max_iter": 1000, "tol": rng.choice([1e-6, 1e-9]), "plan": rng.random() < 0.5, "grad": False}
    if kind == "grad":
        return {"kind": rng.choice(["vanilla", "log"]), "m": _log_int(rng, 64, 2500), "n": _log_int(rng, 64, 2500),
                "d": rng.choice([2, 3, 64]), "alpha": 1.0, "reg": rng.choice([0.05, 0.1]),
                "max_iter": rng.choice([20, 50, 100]), "tol": 0.0, "plan": False, "grad": True}
    if kind == "bary":
        return {"kind": "bary", "log": rng.random() < 0.5, "m": _log_int(rng, 64, 2048), "n": _log_int(rng, 64, 2048),
                "s": _log_int(rng, 2, 40), "d": rng.choice([2, 50]), "reg": rng.choice([0.05, 0.1]),
                "max_iter": rng.choice([20, 50]), "tol": rng.choice([0.0, 1e-6]), "grad": rng.random() < 0.5}
    if kind == "sharp":
        n = _log_int(rng, 64, 512)
        return {"kind": "bary", "log": True, "m": n, "n": n, "s": _log_int(rng, 2, 12), "d": 2, "reg": 0.001,
                "max_iter": 20, "tol": 0.0, "grad": rng.random() < 0.5}
    if kind == "wdl":
        return {"kind": "wdl", "n": _log_int(rng, 200, 5000), "s": rng.choice([4, 6, 10, 16, 20]),
                "docs": rng.choice([16, 31, 48]), "d": 64, "reg": rng.choice([0.05, 0.1]), "max_iter": rng.choice([10, 20])}
    if kind == "train":
        return {"kind": "train", "n": _log_int(rng, 100, 1500), "s": rng.choice([4, 6, 10]), "docs": _log_int(rng, 32, 160),
                "batch": rng.choice([16, 32, 64]), "d": 64, "reg": rng.choice([0.05, 0.1]), "max_iter": rng.choice([10, 20])}
    return {"kind": "stream", "count": _log_int(rng, 6, 100), "lo": 64, "hi": rng.choice([512, 2048, 4096]),
            "max_iter": 2000, "tol": rng.choice([1e-6, 1e-9])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _dirichlet(gen, alpha, *shape):
    """Dirichlet(alpha) draws along the last axis."""
    x = torch._standard_gamma(torch.full(shape, alpha, dtype=F64, device=DEV), generator=gen)
    return x / x.sum(-1, keepdim=True)


def _cost(x, y):
    """Squared Euclidean distances over their maximum, as an (n, m) tensor: the
    m x n cost of sources x, targets y in column-major order."""
    c = (y * y).sum(1)[:, None] + (x * x).sum(1)[None, :]
    c -= 2.0 * (y @ x.T)
    c.clamp_(min=0.0)
    return c / c.max()


def _points(gen, n, d):
    """Uniform points in the unit cube for low dimensions, Gaussian embeddings otherwise."""
    if d <= 3:
        return torch.rand((n, d), dtype=F64, device=DEV, generator=gen)
    return torch.randn((n, d), dtype=F64, device=DEV, generator=gen)


def _sinkhorn_inputs(case, seed):
    g = _gen(seed)
    a = _dirichlet(g, case["alpha"], case["m"])
    b = _dirichlet(g, case["alpha"], case["n"])
    C = _cost(_points(g, case["m"], case["d"]), _points(g, case["n"], case["d"]))
    return a, b, C


def _bary_inputs(case, seed):
    """A (s, m), w (s), C (n, m), b_ext (n): column-major m x s, m x n."""
    g = _gen(seed)
    x = _points(g, case["m"], case["d"])
    y = x if case["n"] == case["m"] else _points(g, case["n"], case["d"])
    # sharp plans: keep every mass well above the plan's smallest entries
    A = _dirichlet(g, 0.3 if case["reg"] > 0.01 else 2.0, case["s"], case["m"])
    w = _dirichlet(g, 1.0, case["s"])
    b = _dirichlet(g, 0.3, case["n"])
    return A, w, _cost(x, y), b


def _documents(gen, n, count):
    """(count, n) word frequencies: 20 to 200 tokens each, Zipf(1.1) word ids."""
    p = torch.arange(1, n + 1, dtype=F64, device=DEV) ** -1.1
    ids = torch.multinomial(p.expand(count, n), 200, replacement=True, generator=gen)
    length = torch.randint(20, 201, (count, 1), device=DEV, generator=gen)
    keep = (torch.arange(200, device=DEV)[None, :] < length).to(F64)
    y = torch.zeros((count, n), dtype=F64, device=DEV).scatter_add_(1, ids, keep)
    return y / y.sum(1, keepdim=True)


def _wdl_inputs(case, seed):
    """Topics A (s, n), weights W (docs, s), documents Y (docs, n), cost C (n, n)."""
    g = _gen(seed)
    x = _points(g, case["n"], case["d"])
    C = _cost(x, x)
    Y = _documents(g, case["n"], case["docs"])
    alpha = 0.1 * torch.randn((case["s"], case["n"]), dtype=F64, device=DEV, generator=g)
    lam = 0.1 * torch.randn((case["docs"], case["s"]), dtype=F64, device=DEV, generator=g)
    return alpha, lam, Y, C


def _requests(case, seed):
    """Sizes, regularisation and data of the stream's requests.  The largest
    and smallest size are fixed, so that every seed asks for about the same work."""
    rs = np.random.default_rng(1234 + case["count"])  # the mix is part of the case
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    g = _gen(seed)
    out = []
    for _ in range(case["count"]):
        m, n = (int(round(math.exp(rs.uniform(lo, hi)))) for _ in range(2))
        d, reg = int(rs.choice([2, 3, 64])), float(rs.choice([0.01, 0.05, 0.1]))
        x = torch.rand((m, d), dtype=F64, device=DEV, generator=g)
        y = torch.rand((n, d), dtype=F64, device=DEV, generator=g)
        out.append((_dirichlet(g, 1.0, m), _dirichlet(g, 1.0, n), _cost(x, y), reg))
    return out


def _empty(*shape):
    return torch.empty(shape, dtype=F64, device=DEV)


def _vp(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k in ("vanilla", "log"):
        m, n = case["m"], case["n"]
        s["a"], s["b"], s["C"] = _sinkhorn_inputs(case, seed)
        s["x"], s["y"] = _empty(m), _empty(n)
        s["P"] = _empty(n, m) if case["plan"] else None
        s["grad_a"] = _empty(m) if case["grad"] else None
    elif k == "host":
        a, b, C = _sinkhorn_inputs(case, seed)
        s["a"], s["b"], s["C"] = a.cpu().numpy(), b.cpu().numpy(), np.asfortranarray(C.cpu().numpy().T)
    elif k == "bary":
        m, n, S = case["m"], case["n"], case["s"]
        s["A"], s["w"], s["C"], s["b_ext"] = _bary_inputs(case, seed)
        s["x1"], s["x2"], s["b"] = _empty(S, m), _empty(S, n), _empty(n)
        s["grad_A"], s["grad_w"] = (_empty(S, m), _empty(S)) if case["grad"] else (None, None)
    elif k == "wdl":
        alpha, lam, s["Y"], s["C"] = _wdl_inputs(case, seed)
        s["A"], s["W"] = torch.softmax(alpha, 1), torch.softmax(lam, 1)
        s["g_alpha"], s["g_lambda"] = _empty(case["s"], case["n"]), _empty(case["s"])
    elif k == "train":
        alpha, lam, Y, C = _wdl_inputs(case, seed)
        for name, t in (("alpha", alpha), ("lam", lam), ("Y", Y), ("C", C)):
            s[name] = np.asfortranarray(t.cpu().numpy().T)
    elif k == "stream":
        reqs = _requests(case, seed)
        s["reqs"] = reqs
        s["f"], s["g"] = _empty(sum(len(r[0]) for r in reqs)), _empty(sum(len(r[1]) for r in reqs))
        arr = (_lib.Problem * len(reqs))()
        at = [0, 0]
        for i, (a, b, C, reg) in enumerate(reqs):
            arr[i] = _lib.Problem(_vp(a), _vp(b), _vp(C), len(a), len(b), reg, case["max_iter"], case["tol"], None,
                                  _vp(s["f"][at[0]:]), _vp(s["g"][at[1]:]))
            at = [at[0] + len(a), at[1] + len(b)]
        s["problems"], s["results"] = arr, (_lib.Result * len(reqs))()
    else:
        raise ValueError(k)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    s, case = state, state["case"]
    k = case["kind"]
    if k == "vanilla":
        r = rw.sinkhorn_vanilla_device(s["a"], s["b"], s["C"], case["reg"], case["max_iter"], case["tol"], P=s["P"],
                                       u=s["x"], v=s["y"], grad_a=s["grad_a"])
        return {"u": s["x"], "v": s["y"], "P": s["P"], "grad_a": s["grad_a"], "loss": r["loss"], "iter": r["iter"]}
    if k == "log":
        r = rw.sinkhorn_log_device(s["a"], s["b"], s["C"], case["reg"], case["max_iter"], case["tol"], P=s["P"],
                                   f=s["x"], g=s["y"], grad_a=s["grad_a"])
        return {"f": s["x"], "g": s["y"], "P": s["P"], "grad_a": s["grad_a"], "loss": r["loss"], "iter": r["iter"]}
    if k == "host":
        r = rw.sinkhorn(s["a"], s["b"], s["C"], {"reg": case["reg"], "max_iter": case["max_iter"], "zero_tol": case["tol"]})
        x, y = ("f", "g") if r["method"] == "log" else ("u", "v")
        return {"x": r[x], "y": r[y], "P": r["P"], "loss": r["loss"], "iter": r["iter"]}
    if k == "bary":
        lib = rw.load()
        fn = lib.rwig_barycenter_log_dev if case["log"] else lib.rwig_barycenter_parallel_dev
        loss, err, it = ctypes.c_double(), ctypes.c_double(), ctypes.c_int()
        _lib.check(fn(_vp(s["x1"]), _vp(s["x2"]), _vp(s["b"]), _vp(s["grad_A"]), _vp(s["grad_w"]), ctypes.byref(loss),
                      ctypes.byref(it), ctypes.byref(err), _vp(s["A"]), _vp(s["w"]), _vp(s["C"]), _vp(s["b_ext"]),
                      case["m"], case["n"], case["s"], case["reg"], int(case["grad"]), case["max_iter"], case["tol"], None))
        out = {"x1": s["x1"], "x2": s["x2"], "b": s["b"], "iter": it.value}
        if case["grad"]:
            out.update(grad_A=s["grad_A"], grad_w=s["grad_w"], loss=loss.value)
        return out
    if k == "wdl":
        _lib.check(rw.load().rwig_wdl_batch_grad_dev(_vp(s["g_alpha"]), _vp(s["g_lambda"]), _vp(s["A"]), _vp(s["W"]),
                                                     _vp(s["Y"]), _vp(s["C"]), case["n"], case["s"], case["docs"],
                                                     case["reg"], case["max_iter"], 1, None))
        return {"g_alpha": s["g_alpha"], "g_lambda": s["g_lambda"]}
    if k == "train":
        return rw.wdl_cpp(s["Y"], s["C"], case["reg"], case["s"], case["batch"], 1, max_iter=case["max_iter"],
                          zero_tol=1e-6, Alpha0=s["alpha"], Lambda0=s["lam"])
    if k == "stream":
        _lib.check(rw.load().rwig_batch_sinkhorn_log_dev(s["problems"], len(s["results"]), s["results"], None))
        return {"f": s["f"], "g": s["g"], "loss": np.array([r.loss for r in s["results"]]),
                "iter": np.array([r.iter for r in s["results"]])}
    raise ValueError(k)


# ---------------------------------------------------------------------------
# work of a pass
# ---------------------------------------------------------------------------
def _iters(reg, tol, max_iter):
    """About how many iterations a solve takes on such inputs (all of them without a stopping test)."""
    if tol <= 0.0:
        return max_iter
    return min(max_iter, int((2.0 if reg >= 0.1 else 4.0 if reg >= 0.05 else 24.0) * -math.log10(tol)))


def work(case):
    k = case["kind"]
    if k in ("vanilla", "log", "host"):
        m, n = case["m"], case["n"]
        it = _iters(case["reg"], case["tol"], case["max_iter"])
        plan, grad = case.get("plan", True), case.get("grad", False)
        return {"bytes": 8.0 * (m * n * (2 if plan else 1) + 2 * (m + n) + (m if grad else 0)),
                "flops": 4.0 * m * n * it * (2 if grad else 1)}
    if k == "bary":
        m, n, S = case["m"], case["n"], case["s"]
        it = _iters(case["reg"], case["tol"], case["max_iter"]) if case["tol"] > 0 else case["max_iter"]
        vec = 2 * m * S + n * S + n + S + (m * S + S + n if case["grad"] else 0)
        return {"bytes": 8.0 * (m * n + vec), "flops": 2.0 * m * n * S * (2 * it * (2 if case["grad"] else 1) + 1)}
    if k in ("wdl", "train"):
        n, S, D, it = case["n"], case["s"], case["docs"], case["max_iter"]
        train = k == "train"
        return {"bytes": 8.0 * (n * n + (2 if train else 1) * n * D + 2 * n * S + 2 * S * D),
                "flops": 2.0 * n * n * S * D * ((4 * it - 1) + (2 * it + 1 if train else 0))}
    rs = np.random.default_rng(1234 + case["count"])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    nbytes = flops = 0.0
    for _ in range(case["count"]):
        m, n = (int(round(math.exp(rs.uniform(lo, hi)))) for _ in range(2))
        _, reg = rs.choice([2, 3, 64]), float(rs.choice([0.01, 0.05, 0.1]))
        nbytes += 8.0 * (m * n + 2 * (m + n))
        flops += 4.0 * m * n * _iters(reg, case["tol"], case["max_iter"])
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain float64 torch
# ---------------------------------------------------------------------------
def _sinkhorn_exact(a, b, C, reg, max_iter, tol, log, grad):
    """u, v, plan, loss, iterations and d loss / d a; C is (n, m)."""
    K = torch.exp(-C / reg)
    a = a.clone().requires_grad_(grad)
    v = torch.ones_like(b)
    Kv = K.T @ v
    it, err = 0, 1000.0
    u = torch.ones_like(a)
    while it < max_iter and err >= tol:
        it += 1
        u = a / Kv
        KTu = K @ u
        v = b / KTu
        Kv = K.T @ v
        if tol > 0.0:
            with torch.no_grad():
                if log:
                    e1, e2 = torch.log(u * Kv) - torch.log(a), torch.log(v * KTu) - torch.log(b)
                else:
                    e1, e2 = u * Kv - a, v * KTu - b
                err = float(e1.norm() + e2.norm())
    P = torch.exp((reg * torch.log(u)[None, :] + reg * torch.log(v)[:, None] - C) / reg)
    loss = (C * P).sum() + reg * (P * (torch.log(P) - 1.0)).sum()
    ga = torch.autograd.grad(loss, a)[0] if grad else None
    return u.detach(), v.detach(), P.detach(), float(loss.detach()), it, ga


def _bary_exact(case, seed):
    """Scaling form where exp(-C/reg) allows it, soft-mins in the log domain otherwise."""
    A, w, C, b_ext = _bary_inputs(case, seed)
    reg, log, grad, tol = case["reg"], case["log"], case["grad"], case["tol"]
    A.requires_grad_(grad)
    w.requires_grad_(grad)
    sharp = float(C.max()) / reg > 600.0
    lk = -C / reg
    K = None if sharp else torch.exp(lk)
    logA = torch.log(A)

    def rows(lv):  # log sum_j K_ij exp(lv_sj), as (s, m)
        return torch.stack([torch.logsumexp(lk + x[:, None], 0) for x in lv]) if sharp else torch.log(torch.exp(lv) @ K)

    def cols(lu):  # log sum_i K_ij exp(lu_si), as (s, n)
        return torch.stack([torch.logsumexp(lk + x[None, :], 1) for x in lu]) if sharp else torch.log(torch.exp(lu) @ K.T)

    it, err = 0, 1000.0
    lv = torch.zeros((case["s"], case["n"]), dtype=F64, device=DEV)
    ly = rows(lv)
    while it < case["max_iter"] and err >= tol:
        it += 1
        lu = logA - ly
        lz = cols(lu)
        lb = (w[:, None] * lz).sum(0)
        lv = lb[None, :] - lz
        ly = rows(lv)
        if tol > 0.0:
            with torch.no_grad():
                D = (lu + ly - logA) if log else torch.exp(lu + ly) - A
                err = float(torch.linalg.matrix_norm(D, 2) if log else D.norm())
    b = torch.exp(lb)
    bn = (b / b.sum()).detach()
    x1, x2 = (reg * lu, reg * lv) if log else (torch.exp(lu), torch.exp(lv))
    out = {"x1": x1.detach(), "x2": x2.detach(), "b": bn, "iter": it}
    if grad:
        # the log form differentiates log b with the normalised b held in its seed
        goal = ((2.0 * (bn - b_ext) * bn) * lb).sum() if log else ((b - b_ext) ** 2).sum()
        out["grad_A"], out["grad_w"] = torch.autograd.grad(goal, (A, w))
        out["loss"] = float(((bn - b_ext) ** 2).sum())
    return out


def _wdl_forward(A, W, K, L):
    """The documents' un-normalised barycenters (docs, n) after L iterations."""
    D, S = W.shape
    v = torch.ones((D, S, K.shape[0]), dtype=F64, device=DEV)
    for _ in range(L):
        u = A[None] / (v @ K)
        z = u @ K.T
        b = torch.exp((W[:, :, None] * torch.log(z)).sum(1))
        v = b[:, None, :] / z
    return b


def _wdl_grad(A, W, Y, K, L):
    """Batch-mean gradients with respect to the logits of A and W."""
    A, W = A.detach().requires_grad_(True), W.detach().requires_grad_(True)
    gA, gW = torch.autograd.grad(((_wdl_forward(A, W, K, L) - Y) ** 2).sum(), (A, W))
    A, W, D = A.detach(), W.detach(), len(Y)
    gA = A * (gA - (A * gA).sum(1, keepdim=True)) / D
    return gA, (W * (gW - (W * gW).sum(1, keepdim=True))).mean(0)


def _train_exact(case, seed):
    al, la, Y, C = _wdl_inputs(case, seed)
    K = torch.exp(-C / case["reg"])
    m = [torch.zeros_like(al), torch.zeros_like(la)]
    v = [torch.zeros_like(al), torch.zeros_like(la)]
    for step, b0 in enumerate(range(0, case["docs"], case["batch"]), 1):
        sl = slice(b0, b0 + case["batch"])
        gA, gl = _wdl_grad(torch.softmax(al, 1), torch.softmax(la, 1)[sl], Y[sl], K, case["max_iter"])
        for x, g, mm, vv in ((al, gA, m[0], v[0]), (la, gl.expand_as(la), m[1], v[1])):  # AdamW
            mm.mul_(0.9).add_(g, alpha=1.0 - 0.9)
            vv.mul_(0.999).add_(g * g, alpha=1.0 - 0.999)
            x.mul_(1.0 - 0.001 * 0.01).sub_(0.001 * (mm / (1 - 0.9 ** step)) / ((vv / (1 - 0.999 ** step)).sqrt() + 1e-8))
    A, W = torch.softmax(al, 1), torch.softmax(la, 1)
    yhat = []
    for w in W:  # each document's barycenter with its own stopping test
        vv = torch.ones_like(A)
        kv, it, err = vv @ K, 0, 1000.0
        while it < case["max_iter"] and err >= 1e-6:
            it += 1
            u = A / kv
            z = u @ K.T
            b = torch.exp((w[:, None] * torch.log(z)).sum(0))
            vv = b[None] / z
            kv = vv @ K
            err = float((u * kv - A).norm())
        yhat.append(b / b.sum())
    return {"A": A.T.contiguous(), "W": W.T.contiguous(), "Yhat": torch.stack(yhat).T.contiguous()}


def exact(case, seed):
    k = case["kind"]
    if k in ("vanilla", "log", "host"):
        a, b, C = _sinkhorn_inputs(case, seed)
        log = k == "log"
        if k == "host":
            log = rw.choose_sinkhorn_method(C.cpu().numpy(), case["reg"], 0.1) == "log"
        u, v, P, loss, it, ga = _sinkhorn_exact(a, b, C, case["reg"], case["max_iter"], case["tol"], log,
                                                case.get("grad", False))
        x, y = (case["reg"] * torch.log(u), case["reg"] * torch.log(v)) if log else (u, v)
        if k == "host":
            return {"x": x, "y": y, "P": P.T.contiguous(), "loss": loss, "iter": it}
        n1, n2 = ("f", "g") if log else ("u", "v")
        return {n1: x, n2: y, "P": P if case["plan"] else None, "grad_a": ga, "loss": loss, "iter": it}
    if k == "bary":
        return _bary_exact(case, seed)
    if k == "wdl":
        alpha, lam, Y, C = _wdl_inputs(case, seed)
        gA, gl = _wdl_grad(torch.softmax(alpha, 1), torch.softmax(lam, 1), Y, torch.exp(-C / case["reg"]), case["max_iter"])
        return {"g_alpha": gA, "g_lambda": gl}
    if k == "train":
        return _train_exact(case, seed)
    out = {"f": [], "g": [], "loss": [], "iter": []}
    for a, b, C, reg in _requests(case, seed):
        u, v, _, loss, it, _ = _sinkhorn_exact(a, b, C, reg, case["max_iter"], case["tol"], True, False)
        out["f"].append(reg * torch.log(u))
        out["g"].append(reg * torch.log(v))
        out["loss"].append(loss)
        out["iter"].append(it)
    return {"f": torch.cat(out["f"]), "g": torch.cat(out["g"]), "loss": np.array(out["loss"]), "iter": np.array(out["iter"])}
