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
