"""The coarsest level's sweeps in one cluster against a launch per sweep
(GB_EXACT_CTAS=0): one multigrid cycle each, on coarsest levels just above the
1024 rows of the dense maps, with one and several slices per CTA, with long
rows (Q2), transposed, from a non-zero start (the second visit of a W cycle),
with the fewest sweeps it takes, and on a level that does not fit.

Both sum the same products in another order: a row of at most 125 terms is off
by at most 125 roundings of its largest partial sum, and ten damped sweeps and
the transfers add at most a factor of ten: 125 * 10 * 1.1e-16 in FP64 and
125 * 10 * 6e-8 in FP32, relative to the result's largest value."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import seeded_inputs, structured_problem, structured_q2

pytestmark = pytest.mark.gpu


def _q1(dim, coarse, beta=None):
    return structured_problem(dim, coarse, 2, *seeded_inputs(dim, coarse, 2), beta=beta)


CASES = {
    "q1_2d_1225": lambda: _q1(2, 17),
    "q1_3d_1331": lambda: _q1(3, 5, (1.0, 0.5, 0.25)),
    "q1_3d_3375": lambda: _q1(3, 7),
    "q1_3d_9261": lambda: _q1(3, 10),  # FP64: too large for the shared memory
    "q2_3d_1331": lambda: structured_q2(3, 5, 2),
}


def _cycles(prob, ctas, **keys):
    old = os.environ.get("GB_EXACT_CTAS")
    if ctas is not None:
        os.environ["GB_EXACT_CTAS"] = ctas
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_EXACT_CTAS", None)
        if old is not None:
            os.environ["GB_EXACT_CTAS"] = old
    out = []
    with ctx:
        ctx.load_problem(prob)
        fine = prob.nlevels - 1
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(fine, y, prob.rhs)
        for transposed in (0, 1):
            ctx.set_operator(transposed)
            ctx.set_params(omega=0.4, **keys)
            for precision in (GB_FP64, GB_FP32):
                ctx.zero(fine, x)
                ctx.precondition(x, y, precision)
                out.append((precision, ctx.download(fine, x)))
    return out


@pytest.mark.parametrize("keys", [dict(), dict(mgtype="W"), dict(iterexact=3),
                                  dict(iterexact=2, iterpre=0)],
                         ids=["v", "w", "three", "two"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_exact_sweeps_equal_launches(name, keys):
    prob = CASES[name]()
    for (prec, a), (_, b) in zip(_cycles(prob, None, **keys), _cycles(prob, "0", **keys)):
        unit = 6e-8 if prec == GB_FP32 else 1.1e-16
        assert np.abs(a - b).max() <= 1250 * unit * np.abs(b).max()
