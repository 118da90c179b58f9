"""Per-kernel times (gb_set_timing) of the left-preconditioned solve: every
repeated solve is timed, not only the ones before its graph exists."""
import pytest

from gascoignelib_b200.native import Context
from gascoignelib_b200.problem import structured_problem

pytestmark = pytest.mark.gpu


def test_repeated_left_solves_are_timed():
    P = structured_problem(2, 2, 4)
    with Context(0) as ctx:
        ctx.load_problem(P)
        ctx.set_params(gmressize=21, tol=1e-8, globaltol=1e-300, maxiter=20)
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(P.nlevels - 1, y, P.rhs)
        steps = [ctx.gmres(x, y)["iterations"] for _ in range(3)]
        counts = []
        for _ in range(3):
            ctx.set_timing(True)
            steps.append(ctx.gmres(x, y)["iterations"])
            times = ctx.kernel_times()
            counts.append(sum(n for name, (n, _) in times.items() if "k_cgs" in name))
        ctx.set_timing(False)
        steps.append(ctx.gmres(x, y)["iterations"])
        assert len(set(steps)) == 1
        assert counts == [2 * steps[0]] * 3
