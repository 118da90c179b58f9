"""The left-preconditioned solver as one graph (CGS2, gmressize up to 32) against
the oracle's modified Gram-Schmidt and against the host-driven path: the
smallest and largest basis of the graph, the first size that keeps the host
path, a right-hand side of zero, and the graph against the same steps launched
by the host, bit for bit.

A few steps are compared before convergence: both bases span the same space and
are orthogonal to rounding, so the iterates differ by roundings of the cycle
(1e-11, the tests' bound for one FP64 cycle) times the few steps."""
import os

import numpy as np
import pytest

from _util import rel_l2
from gascoignelib_b200.native import Context
from gascoignelib_b200.problem import seeded_inputs, structured_problem
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
KEYS = dict(iterpre=2, iterpost=2, iterexact=10, omega=0.8)


def _problem():
    return structured_problem(2, 3, 3, *seeded_inputs(2, 3, 3), beta=(1.0, 0.5))


def _solve(prob, rhs, vmax, graph=None, **keys):
    old = os.environ.get("GB_GRAPH")
    if graph is not None:
        os.environ["GB_GRAPH"] = graph
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_GRAPH", None)
        if old is not None:
            os.environ["GB_GRAPH"] = old
    with ctx:
        ctx.load_problem(prob)
        ctx.set_params(**KEYS, gmressize=vmax, maxiter=100, globaltol=1e-300, **keys)
        fine = prob.nlevels - 1
        x, b = ctx.vec(), ctx.vec()
        ctx.upload(fine, b, rhs)
        ctx.gmres(x, b)  # the second solve runs the graph as the first left it
        info = ctx.gmres(x, b)
        return ctx.download(fine, x), info


@pytest.mark.parametrize("vmax,tol", [(2, 1e-30), (3, 1e-30), (6, 1e-30), (32, 1e-10), (33, 1e-10)])
def test_left_solver_against_oracle(vmax, tol):
    P = _problem()
    u, info = _solve(P, P.rhs, vmax, tol=tol)
    uo, io = Oracle(P, **KEYS).gmres(vmax=vmax, tol=tol, globaltol=1e-300)
    assert info["iterations"] == io["iterations"]
    assert info["status_name"] == ("converged" if tol > 1e-20 else "running")
    assert rel_l2(u, uo) < 1e-10


def test_left_solver_graph_equals_launches():
    P = _problem()
    a, ia = _solve(P, P.rhs, 21, graph="1", tol=1e-10)
    b, ib = _solve(P, P.rhs, 21, graph="0", tol=1e-10)
    assert np.array_equal(a, b)
    for key in ("iterations", "status", "residual", "firstresidual", "kernel_launches"):
        assert ia[key] == ib[key], key


def test_left_solver_zero_right_hand_side():
    P = _problem()
    for graph in ("1", "0"):
        u, info = _solve(P, np.zeros_like(P.rhs), 21, graph=graph, tol=1e-10)
        assert not u.any() and info["iterations"] == 0 and info["status_name"] == "converged"
