"""Which coarsest levels' sweeps run in one cluster, told by the launches of a cycle:
fewer than with a launch per sweep (GB_EXACT_CTAS=0) below the rule's line for a row
length and precision, the same above it and on the long rows of quadratic elements
(there the same kernels run: the same bits).

The results differ by the order of a row's sum: at most 125 terms, ten damped sweeps
and the transfers, 125 * 10 roundings of the result's largest value."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import seeded_inputs, structured_problem, structured_q2

pytestmark = pytest.mark.gpu


def _cycle(prob, ctas, precision):
    old = os.environ.pop("GB_EXACT_CTAS", None)
    if ctas is not None:
        os.environ["GB_EXACT_CTAS"] = ctas
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_EXACT_CTAS", None)
        if old is not None:
            os.environ["GB_EXACT_CTAS"] = old
    with ctx:
        ctx.load_problem(prob)
        ctx.set_params(omega=0.4)
        fine = prob.nlevels - 1
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(fine, y, prob.rhs)
        ctx.precondition(x, y, precision)
        ctx.zero(fine, x)
        before = ctx.kernel_count()
        ctx.precondition(x, y, precision)
        return ctx.kernel_count() - before, ctx.download(fine, x)


def _q1(dim, coarse):
    return structured_problem(dim, coarse, 2, *seeded_inputs(dim, coarse, 2))


# coarsest rows: 1,681 and 2,401; 2,197, 3,375 and 4,913; 1,225; 1,331 and 2,197
@pytest.mark.parametrize("name,prob,in_cluster", [
    ("q1_2d_1681", lambda: _q1(2, 20), (True, True)),
    ("q1_2d_2401", lambda: _q1(2, 24), (False, False)),
    ("q1_3d_2197", lambda: _q1(3, 6), (True, True)),
    ("q1_3d_3375", lambda: _q1(3, 7), (False, True)),
    ("q1_3d_4913", lambda: _q1(3, 8), (False, False)),
    ("q2_2d_1225", lambda: structured_q2(2, 17, 2), (False, False)),
    ("q2_3d_1331", lambda: structured_q2(3, 5, 2), (False, False)),
    ("q2_3d_2197", lambda: structured_q2(3, 6, 2), (False, False)),
])
def test_rule(name, prob, in_cluster):
    P = prob()
    for precision, expected in zip((GB_FP64, GB_FP32), in_cluster):
        fewer, a = _cycle(P, None, precision)
        each, b = _cycle(P, "0", precision)
        assert (fewer < each - 5) == expected
        assert expected or (fewer == each and np.array_equal(a, b))
        unit = 6e-8 if precision == GB_FP32 else 1.1e-16
        assert np.abs(a - b).max() <= 1250 * unit * np.abs(b).max()
