"""A wait that runs out while a context forms its coarse-level maps (the first
cycle: one substitution per unit vector) leaves no trace in them: after the
GB_ETIMEOUT the same context gives the same bits as one that never timed out."""
import numpy as np
import pytest

from gascoignelib_b200.native import GB_ETIMEOUT, GB_FP32, GB_FP64, Context, GBError, lib
from gascoignelib_b200.problem import seeded_inputs, structured_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [GB_FP64, GB_FP32])
@pytest.mark.parametrize("call", ["precondition", "fgmres"])
def test_maps_are_formed_again(call, precision):
    P = structured_problem(2, 2, 5, *seeded_inputs(2, 2, 5))
    fine = P.nlevels - 1
    results = []
    for bad_start in (False, True):
        with Context(0) as ctx:
            ctx.load_problem(P)
            ctx.set_params(gmressize=21, tol=1e-8, globaltol=1e-300, maxiter=20, omega=0.8,
                           smoother="ilu")
            x, y = ctx.vec(), ctx.vec()
            ctx.upload(fine, y, P.rhs)

            def run():
                ctx.zero(fine, x)
                if call == "precondition":
                    ctx.precondition(x, y, precision)
                else:
                    ctx.fgmres(x, y, precision, check=False)
                return ctx.download(fine, x)

            if bad_start:
                assert lib().gb_set_wait_limit(ctx.h, 1_000_000, 1) == 0
                with pytest.raises(GBError) as e:
                    run()
                assert e.value.code == GB_ETIMEOUT
                assert lib().gb_set_wait_limit(ctx.h, 1_000_000_000, 0) == 0
            results += [run(), run()]
    assert np.isfinite(results[0]).all()
    for r in results[1:]:
        assert np.array_equal(r, results[0])
