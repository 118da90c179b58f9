"""gb_set_wait_limit bounds each wait of the block ILU's substitution cluster, not
the time of a whole substitution: a chain of 20,000 rows, each of which waits for
the one before it for well below a microsecond, runs for milliseconds under a
limit of 0.3 ms. A wait that does run out ends the call with GB_ETIMEOUT, and the
context stays usable."""
import numpy as np
import pytest

from gascoignelib_b200.native import GB_ETIMEOUT, GB_FP32, Context, GBError, lib
from gascoignelib_b200.problem import Level, Problem, seeded_inputs, structured_problem

pytestmark = pytest.mark.gpu


def _chain(n):
    """One level: a tridiagonal matrix, whose ILU is its exact LU."""
    rng = np.random.default_rng(3)
    i = np.arange(n)
    rows = np.stack([i - 1, i, i + 1], axis=1)
    keep = (rows >= 0) & (rows < n)
    ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    col = rows[keep].astype(np.int64)
    diag = (ptr[:-1] + (i > 0)).astype(np.int64)
    val = rng.uniform(-1.0, 1.0, col.size)
    val[diag] = 4.0
    level = Level(n=n, B=1, rowptr=ptr, col=col, diag=diag, val=val,
                  dirichlet=np.array([], dtype=np.int64))
    return Problem(dim=2, levels=[level], transfers=[], rhs=rng.uniform(-1, 1, n))


def test_limit_bounds_one_wait():
    P = _chain(20000)
    with Context(0) as ctx:
        ctx.load_problem(P)
        ctx.set_params(omega=1.0, smoother="ilu")
        assert lib().gb_set_wait_limit(ctx.h, 300_000, 0) == 0
        x, y, h = ctx.vec(), ctx.vec(), ctx.vec()
        ctx.upload(0, y, P.rhs)
        ctx.zero(0, x)
        ctx.smooth(0, 1, x, y, h)
        ctx.residualgmres(0, h, x, y)
        # the factors are exact: one sweep solves the (well conditioned) system
        assert np.abs(ctx.download(0, h)).max() < 1e-13


@pytest.mark.parametrize("dim,coarse,refine", [(2, 2, 4), (3, 1, 5)])
def test_wait_runs_out_and_the_context_recovers(dim, coarse, refine):
    # one CTA, and a cluster of several
    P = structured_problem(dim, coarse, refine, *seeded_inputs(dim, coarse, refine))
    with Context(0) as ctx:
        ctx.load_problem(P)
        ctx.set_params(gmressize=21, tol=1e-8, globaltol=1e-300, maxiter=20, omega=0.8,
                       smoother="ilu")
        x, b = ctx.vec(), ctx.vec()
        ctx.upload(P.nlevels - 1, b, P.rhs)
        ref = ctx.fgmres(x, b, GB_FP32)
        u = ctx.download(P.nlevels - 1, x)
        for solve in (lambda: ctx.fgmres(x, b, GB_FP32, check=False), lambda: ctx.gmres(x, b)):
            # a value that never comes, waited for at most 2 ms
            assert lib().gb_set_wait_limit(ctx.h, 2_000_000, 1) == 0
            with pytest.raises(GBError) as e:
                solve()
            assert e.value.code == GB_ETIMEOUT
            assert lib().gb_set_wait_limit(ctx.h, 1_000_000_000, 0) == 0
            assert ctx.fgmres(x, b, GB_FP32)["iterations"] == ref["iterations"]
            assert np.array_equal(ctx.download(P.nlevels - 1, x), u)
