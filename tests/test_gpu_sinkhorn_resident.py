"""Solves that run whole in one launch with the kernel matrix on the chip
(sinkhorn_resident.cu) at the edges of their blocks, against the CPU oracle and
against the general drivers, and the calls they hand back."""
import numpy as np
import pytest

import oracle
import rwig_b200 as rw
from rwig_b200 import synth
from tests.util import PARITY_TOL, dual_scale, rel_err

pytestmark = pytest.mark.gpu

ORACLE = {"vanilla": oracle.sinkhorn_vanilla, "log": oracle.sinkhorn_log}
RESIDENT_LAUNCHES = 2  # the masses and the solve


def _problem(m, n, zeros=False):
    a, b, C = synth.sinkhorn_problem(m, n, 1.0, salt=3 * m + n)
    if zeros:
        a[::3] = 0.0
        b[n // 2:n // 2 + 2] = 0.0
        a, b = a / a.sum(), b / b.sum()
    return a, b, C


def _same(got, ref, reg, method):
    assert got["iter"] == ref["iter"]
    assert got["return_status"] == ref["return_status"]
    assert rel_err(got["P"], ref["P"]) <= PARITY_TOL
    assert abs(got["loss"] - ref["loss"]) <= PARITY_TOL * abs(ref["loss"])
    gs = max(float(np.abs(ref["grad_a"]).max()), abs(ref["loss"]))
    assert rel_err(got["grad_a"], ref["grad_a"], gs) <= PARITY_TOL


# one block and its largest side, one row or column more, thin problems in both
# directions, the most rows, an odd leading dimension, columns in registers (2048)
@pytest.mark.parametrize("m,n,zeros", [
    (3, 2, False), (65, 33, True), (480, 7, False), (481, 480, True), (1, 700, False), (700, 1, False),
    (2, 9000, False), (8192, 3, False), (1223, 1999, True), (2048, 2048, False),
])
@pytest.mark.parametrize("method", ["vanilla", "log"])
def test_blocks(method, m, n, zeros):
    a, b, C = _problem(m, n, zeros)
    par = {"reg": 0.2, "method": method, "with_grad": True, "max_iter": 7, "zero_tol": 1e-13}
    got = rw.sinkhorn(a, b, C, par)
    assert rw.last_report()["kernel_launches"] == RESIDENT_LAUNCHES
    ref = ORACLE[method](a, b, C, 0.2, with_grad=True, max_iter=7, zero_tol=1e-13)
    _same(got, ref, 0.2, method)
    assert rw.last_report()["support_m"] == int((a != 0).sum())


@pytest.mark.parametrize("m,n,reg", [(300, 500, 0.05), (700, 40, 0.01), (150, 1100, 0.004)])
def test_general_path_agrees(m, n, reg):
    """The log method with absorption (log_sinkhorn.tau below its default) runs
    in the general drivers: same iterations, potentials and gradient."""
    a, b, C = _problem(m, n, True)
    par = {"reg": reg, "method": "log", "with_grad": True, "max_iter": 60}
    got = rw.sinkhorn(a, b, C, par)
    resident = rw.last_report()["kernel_launches"]
    L = rw.load()
    L.rwig_set_option(b"log_sinkhorn.tau", 99.0)
    try:
        ref = rw.sinkhorn(a, b, C, par)
    finally:
        L.rwig_set_option(b"log_sinkhorn.tau", 100.0)
    assert resident == RESIDENT_LAUNCHES and rw.last_report()["kernel_launches"] != RESIDENT_LAUNCHES
    _same(got, ref, reg, "log")
    on, om = b != 0.0, a != 0.0
    sc = dual_scale(ref["f"][om], ref["g"][on])
    assert np.abs(got["f"][om] - ref["f"][om]).max() <= PARITY_TOL * sc
    assert np.abs(got["g"][on] - ref["g"][on]).max() <= PARITY_TOL * sc


@pytest.mark.parametrize("reg,grad", [(1e-3, True), (1.4e-3, False)])
def test_handed_back(reg, grad):
    """A kernel matrix with entries below the normal range goes to the general
    drivers; an underflowed plan entry gives the reference's NaN gradient."""
    a, b, C = _problem(90, 70)
    assert C.max() / reg > 709.0
    par = {"reg": reg, "method": "log", "with_grad": grad, "max_iter": 30}
    got = rw.sinkhorn(a, b, C, par)
    assert rw.last_report()["kernel_launches"] != RESIDENT_LAUNCHES
    ref = oracle.sinkhorn_log(a, b, C, reg, with_grad=grad, max_iter=30)
    assert got["iter"] == ref["iter"] and got["return_status"] == ref["return_status"]
    assert rel_err(got["P"], ref["P"]) <= PARITY_TOL
    if grad:
        assert rel_err(got["grad_a"], ref["grad_a"]) <= PARITY_TOL


@pytest.mark.parametrize("narrow", ["a", "b"])
@pytest.mark.parametrize("reg", [0.002, 0.0018, 0.0016])
@pytest.mark.parametrize("method", ["vanilla", "log"])
def test_gradient_of_large_scalings(method, reg, narrow):
    """Sharp kernels (max C / reg from 500 to 625) between a narrow and a broad
    marginal: the scalings pass 1e180, their squares the range of doubles, the
    gradient is of order one."""
    m, n = 60, 70
    g = synth.rng(53, m + n)
    x = g.random((m, 1)) * (0.1 if narrow == "a" else 1.0)
    y = g.random((n, 1)) * (1.0 if narrow == "a" else 0.1)
    C = (x - y.T) ** 2
    C /= C.max()
    a, b = synth.dirichlet(g, 1.0, m), synth.dirichlet(g, 1.0, n)
    got = rw.sinkhorn(a, b, C, {"reg": reg, "method": method, "with_grad": True, "max_iter": 10, "zero_tol": 0.0})
    assert rw.last_report()["kernel_launches"] == RESIDENT_LAUNCHES
    if method == "vanilla":
        assert max(got["u"].max(), got["v"].max()) > 1e155
    ref = ORACLE[method](a, b, C, reg, with_grad=True, max_iter=10, zero_tol=0.0)
    assert np.isfinite(ref["grad_a"]).all()
    _same(got, ref, reg, method)


def test_gradient_history_memory():
    """A gradient keeps each iteration's scalings once, not once per block:
    8 (max_iter + 4)(M + N) bytes, sized by max_iter."""
    import torch
    m, n, max_iter = 600, 500, 5000
    a, b, C = _problem(m, n)
    rw.load().rwig_shutdown()  # start without scratch

    def solve(iters):
        before = torch.cuda.mem_get_info()[0]
        r = rw.sinkhorn(a, b, C, {"reg": 0.2, "method": "log", "with_grad": True, "max_iter": iters})
        assert rw.last_report()["kernel_launches"] == RESIDENT_LAUNCHES and r["iter"] < 100
        return before - torch.cuda.mem_get_info()[0], r

    torch.cuda.mem_get_info()
    _, ref = solve(100)  # the context, module and all other scratch
    grown, got = solve(max_iter)
    # allocations are rounded to 2 MB blocks
    assert grown <= 8 * (max_iter + 4) * (m + n) + 2 * (2 << 20)
    assert np.array_equal(got["grad_a"], ref["grad_a"])


@pytest.mark.parametrize("method", ["vanilla", "log"])
def test_report_of_a_handed_back_call(method):
    """The launches and the time of a solve in one launch that was given up are
    in the report: two launches more than the general drivers alone take."""
    a, b, C = _problem(90, 70)
    a[0] = 1e-280  # its scaling leaves the safe range
    par = {"reg": 0.1, "method": method, "max_iter": 12, "zero_tol": 0.0}
    L = rw.load()
    got = rw.sinkhorn(a, b, C, par)
    back = rw.last_report()
    assert back["iter"] == got["iter"] == 12
    assert back["device_ms"] > back["kernel_ms"]
    if method == "log":
        L.rwig_set_option(b"log_sinkhorn.tau", 99.0)
        try:
            ref = rw.sinkhorn(a, b, C, par)
        finally:
            L.rwig_set_option(b"log_sinkhorn.tau", float("nan"))
        general = rw.last_report()
        assert back["fallback_events"] == general["fallback_events"] + 1  # (it re-runs sweeps of its own)
        assert back["kernel_launches"] == general["kernel_launches"] + RESIDENT_LAUNCHES
        assert rel_err(got["P"], ref["P"]) <= PARITY_TOL
    else:
        assert back["kernel_launches"] > RESIDENT_LAUNCHES and back["fallback_events"] == 1
    assert rel_err(got["P"], ORACLE[method](a, b, C, 0.1, max_iter=12, zero_tol=0.0)["P"]) <= PARITY_TOL


# subnormal entries of K; a plan that underflows from the first iterations on, and
# one that does so on zero entries of K only; a mass whose scaling is out of range;
# a negative one
@pytest.mark.parametrize("m,n,method,reg,mass,zeros", [
    (90, 70, "log", 1e-3, None, False), (481, 300, "log", 1e-3, None, True), (90, 70, "vanilla", 1.2e-3, None, False),
    (200, 300, "vanilla", 1e-3, None, True), (90, 70, "vanilla", 5e-4, None, False), (90, 70, "log", 0.1, 1e-280, True),
    (90, 70, "vanilla", 0.1, 1e-280, False),
])
@pytest.mark.parametrize("max_iter", [1, 2, 3, 25])
def test_handed_back_early(m, n, method, reg, mass, zeros, max_iter):
    """Calls that leave the scaling form in the first iterations or have no
    finite gradient, with full and with reduced supports."""
    a, b, C = _problem(m, n, zeros)
    if mass:
        a[1] = mass
    par = {"reg": reg, "method": method, "with_grad": True, "max_iter": max_iter, "zero_tol": 0.0}
    got = rw.sinkhorn(a, b, C, par)
    rep = rw.last_report()
    assert rep["fallback_events"] >= 1 and rep["kernel_launches"] > RESIDENT_LAUNCHES
    assert rep["support_m"] == int((a != 0).sum()) and rep["support_n"] == int((b != 0).sum())
    ref = ORACLE[method](a, b, C, reg, with_grad=True, max_iter=max_iter, zero_tol=0.0)
    assert got["iter"] == ref["iter"] == max_iter
    assert rel_err(got["P"], ref["P"]) <= PARITY_TOL
    x, y = ("f", "g") if method == "log" else ("u", "v")
    sc = dual_scale(ref[x], ref[y]) if method == "log" else None
    assert rel_err(got[x], ref[x], sc) <= PARITY_TOL and rel_err(got[y], ref[y], sc) <= PARITY_TOL
    if method == "log":
        assert rel_err(got["grad_a"], ref["grad_a"]) <= PARITY_TOL


@pytest.mark.parametrize("m,n", [(2041, 1983), (8190, 479), (600, 6700)])
@pytest.mark.parametrize("max_iter", [1, 2, 6])
def test_gradient_beside_register_columns(m, n, max_iter):
    """Blocks that keep some columns of K in registers fetch the scalings of a
    backward step into shared memory: none for one iteration, one step for two."""
    a, b, C = _problem(m, n, True)
    par = {"reg": 0.2, "method": "log", "with_grad": True, "max_iter": max_iter, "zero_tol": 0.0}
    got = rw.sinkhorn(a, b, C, par)
    assert rw.last_report()["kernel_launches"] == RESIDENT_LAUNCHES
    ref = oracle.sinkhorn_log(a, b, C, 0.2, with_grad=True, max_iter=max_iter, zero_tol=0.0)
    _same(got, ref, 0.2, "log")


@pytest.mark.parametrize("narrow", ["a", "b"])
@pytest.mark.parametrize("method", ["vanilla", "log"])
def test_gradient_of_scalings_out_of_range(method, narrow):
    """Scalings beyond 1e250, which the general drivers take over: the squares
    overflow there too, the gradient does not."""
    m, n, reg = 90, 70, 0.00143
    g = synth.rng(53, m + n)
    x = g.random((m, 1)) * (0.1 if narrow == "a" else 1.0)
    y = g.random((n, 1)) * (1.0 if narrow == "a" else 0.1)
    C = (x - y.T) ** 2
    C /= C.max()
    a, b = synth.dirichlet(g, 1.0, m), synth.dirichlet(g, 1.0, n)
    got = rw.sinkhorn(a, b, C, {"reg": reg, "method": method, "with_grad": True, "max_iter": 10, "zero_tol": 0.0})
    assert rw.last_report()["fallback_events"] >= 1
    ref = ORACLE[method](a, b, C, reg, with_grad=True, max_iter=10, zero_tol=0.0)
    assert np.isfinite(ref["grad_a"]).all()
    _same(got, ref, reg, method)
