"""The coarsest level's sweeps in one cluster, again and again on the same data:
the same bits each time, with several threads sharing a row's sends (small
levels) and with one, on 4, 8 and 16 CTAs, where each sweep's partial sums and
values are read while other CTAs go on to the next."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import seeded_inputs, structured_problem, structured_q2

pytestmark = pytest.mark.gpu

CASES = {
    "q1_2d_1225": lambda: structured_problem(2, 17, 2, *seeded_inputs(2, 17, 2)),
    "q1_3d_3375": lambda: structured_problem(3, 7, 2, *seeded_inputs(3, 7, 2)),
    "q2_3d_1331": lambda: structured_q2(3, 5, 2),
}


@pytest.mark.parametrize("precision", [GB_FP64, GB_FP32])
@pytest.mark.parametrize("ctas", ["4", "8", "16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_repeated_sweeps_give_the_same_bits(name, ctas, precision):
    prob = CASES[name]()
    old = os.environ.get("GB_EXACT_CTAS")
    os.environ["GB_EXACT_CTAS"] = ctas
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_EXACT_CTAS", None)
        if old is not None:
            os.environ["GB_EXACT_CTAS"] = old
    with ctx:
        ctx.load_problem(prob)
        ctx.set_params(omega=0.4, iterexact=20)
        fine = prob.nlevels - 1
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(fine, y, prob.rhs)
        first = None
        for _ in range(60):
            ctx.zero(fine, x)
            ctx.precondition(x, y, precision)
            got = ctx.download(fine, x)
            first = got if first is None else first
            assert np.array_equal(got, first)
