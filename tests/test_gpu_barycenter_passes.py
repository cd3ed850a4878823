"""Soft-min passes of the log-domain barycenter (barycenter_log.cu) at the edges
of a lane's chunk, of the warps along the reduction axis, of the histograms per
warp and of the grid, and problems that move between the two forms."""
import numpy as np
import pytest

import oracle
import rwig_b200 as rw
from rwig_b200 import synth
from tests.util import PARITY_TOL, dual_scale, rel_err

pytestmark = pytest.mark.gpu


def _problem(n, m, S):
    g = synth.rng(43, 7 * n + 3 * m + S)
    C = synth.sq_euclid_cost(g.random((n, 3)), g.random((m, 3)))
    return synth.dirichlet(g, 1.0, n, S), C, synth.dirichlet(g, 1.0, S), synth.dirichlet(g, 1.0, m)


def _check(A, C, w, be, reg, L):
    got = rw.barycenter(A, C, w, be, {"reg": reg, "method": "log", "with_grad": True, "max_iter": L, "zero_tol": 0.0})
    ref = oracle.barycenter_log(A, C, w, be, reg, with_grad=True, max_iter=L, zero_tol=0.0)
    for k in ("b", "F", "G", "grad_A", "grad_w"):
        # a gradient that is zero in exact arithmetic (one histogram, one row)
        # leaves rounding residue of the size of its terms
        sc = dual_scale(ref["F"], ref["G"]) if k in "FG" else float(np.abs(ref[k]).max())
        sc = max(sc, 1.0 if k.startswith("grad") and min(A.shape) == 1 else 0.0)
        assert rel_err(got[k], ref[k], sc) <= PARITY_TOL, k


@pytest.mark.parametrize("n,m,S", [
    (1, 40, 3), (40, 1, 3), (31, 33, 1), (127, 129, 8), (128, 257, 9), (511, 513, 2), (33, 3000, 5), (2600, 70, 16),
])
def test_pass_edges(n, m, S):
    L = rw.load()
    L.rwig_set_option(b"barycenter.log_path", 1.0)
    try:
        _check(*_problem(n, m, S), 0.1, 6)
    finally:
        L.rwig_set_option(b"barycenter.log_path", float("nan"))
    assert rw.last_report()["fallback_events"] == 1


def test_between_the_forms():
    """The same shapes in and out of the scaling form's range in turn, and the
    parallel method, which has no such range, after a call that left it."""
    A, C, w, be = _problem(150, 130, 4)
    for reg, out in ((0.1, 0), (5e-4, 1), (5e-4, 1), (0.1, 0), (0.1, 0), (0.1, 0), (5e-4, 1)):
        _check(A, C, w, be, reg, 5)
        assert rw.last_report()["fallback_events"] == out
    got = rw.barycenter(A, C, w, be, {"reg": 0.1, "method": "parallel", "max_iter": 200, "zero_tol": 1e-8})
    ref = oracle.barycenter_parallel(A, C, w, reg=0.1, max_iter=200, zero_tol=1e-8)
    assert got["iter"] == ref["iter"] and rel_err(got["b"], ref["b"]) <= PARITY_TOL


# kw (warps along the reduction axis) 1, 2 and 4 in both passes, and 4 against 2
EMPTY_SIZES = [(120, 120, 2), (360, 360, 5), (400, 400, 2), (500, 200, 2)]


def _log_path(value):
    rw.load().rwig_set_option(b"barycenter.log_path", value)


@pytest.mark.parametrize("n,m,S", EMPTY_SIZES)
def test_infinite_costs(n, m, S):
    """Forbidden pairs: with a band of finite costs, whole warps of a column or
    a row have no finite term."""
    A, _, w, be = _problem(n, m, S)
    i, j = np.arange(n)[:, None] / n, np.arange(m)[None, :] / m
    C = np.where(np.abs(i - j) <= 15 / max(n, m), (i - j) ** 2, np.inf)
    _log_path(1.0)
    try:
        _check(A, C, w, be, 1e-3, 3)
    finally:
        _log_path(float("nan"))
    _check(A, C, w, be, 1e-3, 3)
    assert rw.last_report()["fallback_events"] == 1


@pytest.mark.parametrize("L", [1, 3])
@pytest.mark.parametrize("n,m,S", EMPTY_SIZES)
def test_zero_mass_runs(n, m, S, L):
    """Histograms supported in 20 neighbouring cells: the zero masses drop out
    of every column's soft-min.  (Their own entries of F are -inf, from the
    second iteration on NaN as in the reference's update.)"""
    A, C, w, be = _problem(n, m, S)
    A[:70] = A[90:] = 0.0
    A /= A.sum(0)
    reg = 0.01
    _log_path(1.0)
    try:
        got = rw.barycenter(A, C, w, be, {"reg": reg, "method": "log", "max_iter": L, "zero_tol": 0.0})
    finally:
        _log_path(float("nan"))
    on = slice(70, 90)
    lk, la = -C[on] / reg, np.log(A[on])

    def lse(x, axis):
        top = x.max(axis, keepdims=True)
        return np.log(np.exp(x - top).sum(axis)) + np.squeeze(top, axis)

    lv = np.zeros((m, S))
    for _ in range(L):
        lu = la - lse(lk[:, :, None] + lv[None], 1)
        lz = lse(lk[:, :, None] + lu[:, None, :], 0)
        lb = lz @ w
        lv = lb[:, None] - lz
    b = np.exp(lb - lb.max())
    assert rel_err(got["b"], b / b.sum()) <= PARITY_TOL
    sc = dual_scale(reg * lu, reg * lv)
    assert rel_err(got["G"], reg * lv, sc) <= PARITY_TOL
    assert rel_err(got["F"][on], reg * lu, sc) <= PARITY_TOL
    if L == 1:
        ref = oracle.barycenter_log(A, C, w, be, reg, max_iter=1, zero_tol=0.0)
        for k in ("b", "F", "G"):
            assert rel_err(got[k], ref[k], None if k == "b" else sc) <= PARITY_TOL, k
