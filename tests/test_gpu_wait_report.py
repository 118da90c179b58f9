"""A device-side wait that runs out is reported by the call that first knows:
a solve, with or without a gb_solve_info; after calls that only enqueue, the
next download or gb_ctx_synchronize. The context stays usable. The waits are
made to run out by arrivals that never come (gb_set_wait_limit's phantoms)."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_ETIMEOUT, GB_FP32, GB_FP64, Context, GBError, lib
from gascoignelib_b200.problem import seeded_inputs, structured_problem

pytestmark = pytest.mark.gpu


@pytest.fixture()
def mid():
    """A context with the multi-CTA cycle, on 33^3 nodes."""
    old = os.environ.get("GB_MID")
    os.environ["GB_MID"] = "1"
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_MID", None)
        if old is not None:
            os.environ["GB_MID"] = old
    with ctx:
        ctx.load_problem(structured_problem(3, 1, 5, *seeded_inputs(3, 1, 5)))
        ctx.set_params(gmressize=21, tol=1e-8, globaltol=1e-300, maxiter=20)
        yield ctx


def _limit(ctx, ns, phantoms):
    assert lib().gb_set_wait_limit(ctx.h, ns, phantoms) == 0


@pytest.mark.parametrize("precision", [GB_FP64, GB_FP32])
@pytest.mark.parametrize("report", ["download", "synchronize"])
def test_cycle_that_only_enqueues(mid, precision, report):
    fine = mid.nlevels - 1
    rhs = np.random.default_rng(1).standard_normal(mid.sizes[fine])
    x, y = mid.vec(), mid.vec()
    mid.upload(fine, y, rhs)

    def cycle():
        mid.zero(fine, x)
        mid.precondition(x, y, precision)
        if report == "synchronize":
            code = lib().gb_ctx_synchronize(mid.h)
            if code:
                raise GBError(code, lib().gb_last_error_string(mid.h).decode())
        return mid.download(fine, x)

    good = cycle()
    _limit(mid, 5_000_000, 1)
    with pytest.raises(GBError) as e:
        cycle()
    assert e.value.code == GB_ETIMEOUT
    assert "grid barrier" in str(e.value)
    _limit(mid, 1_000_000_000, 0)
    assert np.array_equal(cycle(), good)


@pytest.mark.parametrize("method", ["gmres", "fgmres", "solve_host"])
def test_solve_without_info(mid, method):
    fine = mid.nlevels - 1
    rhs = np.random.default_rng(2).standard_normal(mid.sizes[fine])
    x, y = mid.vec(), mid.vec()
    mid.upload(fine, y, rhs)
    L = lib()
    out = np.empty_like(rhs)
    calls = {
        "gmres": lambda: L.gb_gmres(mid.h, x, y, None),
        "fgmres": lambda: L.gb_fgmres(mid.h, x, y, GB_FP32, None),
        "solve_host": lambda: L.gb_solve_host(mid.h, 2, rhs.ctypes.data_as(
            L.gb_solve_host.argtypes[2]), out.ctypes.data_as(L.gb_solve_host.argtypes[3]),
            out.size, None),
    }
    assert calls[method]() == 0
    _limit(mid, 2_000_000, 1)
    assert calls[method]() == GB_ETIMEOUT
    _limit(mid, 1_000_000_000, 0)
    assert calls[method]() == 0
