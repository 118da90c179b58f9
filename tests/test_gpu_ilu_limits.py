"""Levels at the largest size whose FP64 substitutions could fit the cluster's
shared memory, with a row that every CTA uses (no copies of other CTAs' rows): in
FP64 they keep a launch per dependency level, in FP32 they run in the cluster, and
both give the bits of GB_ILU_CTA_ROWS=0."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import Level, Problem

pytestmark = pytest.mark.gpu


def _problem(n, B, far=20000):
    """Rows {0, i - far, i, i + far}: n / far dependency levels."""
    rng = np.random.default_rng(8)
    i = np.arange(n)
    rows = np.stack([0 * i, i - far, i, i + far], axis=1)
    keep = (rows >= 0) & (rows < n)
    keep[:, 0] &= (i != 0) & (i != far)
    ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    col = rows[keep].astype(np.int64)
    diag = ptr[:-1] + keep[:, :2].sum(axis=1)
    val = rng.uniform(-1.0, 1.0, (col.size, B, B))
    val[diag] += 8.0 * np.eye(B)
    level = Level(n=n, B=B, rowptr=ptr, col=col, diag=diag.astype(np.int64), val=val.ravel(),
                  dirichlet=np.array([], dtype=np.int64))
    return Problem(dim=2, levels=[level], transfers=[], rhs=rng.uniform(-1, 1, n * B))


def _results(prob, env):
    old = os.environ.get("GB_ILU_CTA_ROWS")
    os.environ.update(env)
    try:
        ctx = Context(0)
    finally:
        os.environ.pop("GB_ILU_CTA_ROWS", None)
        if old is not None:
            os.environ["GB_ILU_CTA_ROWS"] = old
    with ctx:
        ctx.load_problem(prob)
        ctx.set_params(omega=0.9, smoother="ilu", iterexact=2)
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(0, y, prob.rhs)
        out = []
        for precision in (GB_FP64, GB_FP32):
            ctx.zero(0, x)
            ctx.precondition(x, y, precision)
            out.append(ctx.download(0, x))
        return out


@pytest.mark.parametrize("n,B", [(442368, 1), (442400, 1), (442500, 1), (221200, 2)])
def test_largest_levels(n, B):
    prob = _problem(n, B)
    for a, b in zip(_results(prob, {}), _results(prob, {"GB_ILU_CTA_ROWS": "0"})):
        assert np.isfinite(a).all()
        assert np.array_equal(a, b)


def test_a_long_chain_is_not_packed():
    # 100,000 rows that depend on each other one by one: 5 MB of factors, 820 MB
    # in groups of 32 rows and chunks of 8 entries
    import torch
    n = 100000
    i = np.arange(n)
    rows = np.stack([i - 1, i, i + 1], axis=1)
    keep = (rows >= 0) & (rows < n)
    ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    diag = (ptr[:-1] + (i > 0)).astype(np.int64)
    rng = np.random.default_rng(9)
    val = rng.uniform(-1.0, 1.0, int(ptr[-1]))
    val[diag] = 4.0
    level = Level(n=n, B=1, rowptr=ptr, col=rows[keep].astype(np.int64), diag=diag, val=val,
                  dirichlet=np.array([], dtype=np.int64))
    prob = Problem(dim=2, levels=[level], transfers=[], rhs=rng.uniform(-1, 1, n))
    with Context(0) as ctx:
        ctx.load_problem(prob)
        ctx.set_params(omega=1.0, smoother="ilu")
        x, y, h = ctx.vec(), ctx.vec(), ctx.vec()
        ctx.upload(0, y, prob.rhs)
        ctx.zero(0, x)
        free0, _ = torch.cuda.mem_get_info(0)
        ctx.smooth(0, 1, x, y, h)
        ctx.residualgmres(0, h, x, y)
        assert np.abs(ctx.download(0, h)).max() < 1e-13
        free1, _ = torch.cuda.mem_get_info(0)
        assert free0 - free1 < 200 << 20
