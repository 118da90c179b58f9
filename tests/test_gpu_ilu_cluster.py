"""Both block ILU substitutions in one thread-block cluster against a launch
per dependency level (GB_ILU_CTA_ROWS=0): the same rows' arithmetic in the same
order, so the same bits. Sizes with one row group and with several, one CTA and
sixteen, block sizes 1 to 4, rows longer than one chunk of entries, a Dirichlet
boundary, NaN in the data."""
import os

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64, Context
from gascoignelib_b200.problem import (Level, Problem, seeded_inputs, structured_problem,
                                       structured_q2, structured_stokes)

pytestmark = pytest.mark.gpu


def _diffusion(dim, coarse, refine):
    return structured_problem(dim, coarse, refine, *seeded_inputs(dim, coarse, refine))


def _blocks_of_two(n):
    """One level of 2x2 blocks: a diagonally dominant band matrix with a far entry."""
    rng = np.random.default_rng(5)
    rows = [sorted({j for j in (i - 7, i - 1, i, i + 1, i + 7) if 0 <= j < n}) for i in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    col = np.concatenate(rows).astype(np.int64)
    diag = np.array([ptr[i] + r.index(i) for i, r in enumerate(rows)], dtype=np.int64)
    val = rng.uniform(-1.0, 1.0, size=(col.size, 2, 2))
    val[diag] += 8.0 * np.eye(2)
    level = Level(n=n, B=2, rowptr=ptr, col=col, diag=diag, val=val.ravel(),
                  dirichlet=np.array([0], dtype=np.int64), dircomp_mask=3)
    return Problem(dim=2, levels=[level], transfers=[], rhs=rng.uniform(-1, 1, 2 * n))


def _scattered(n):
    """One level whose rows use rows of many other CTAs (no copies of those then)."""
    rng = np.random.default_rng(6)
    rows = [sorted({i, *rng.integers(0, n, size=5).tolist()}) for i in range(n)]
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    col = np.concatenate(rows).astype(np.int64)
    diag = np.array([ptr[i] + r.index(i) for i, r in enumerate(rows)], dtype=np.int64)
    val = rng.uniform(-1.0, 1.0, size=col.size)
    val[diag] = 8.0
    level = Level(n=n, B=1, rowptr=ptr, col=col, diag=diag, val=val,
                  dirichlet=np.array([0], dtype=np.int64))
    return Problem(dim=2, levels=[level], transfers=[], rhs=rng.uniform(-1, 1, n))


CASES = {
    "2d_4": lambda: _diffusion(2, 2, 1),
    "2d_96": lambda: _diffusion(2, 3, 5),
    "3d_20": lambda: _diffusion(3, 5, 2),
    "3d_48": lambda: _diffusion(3, 3, 4),
    "q2_3d_12": lambda: structured_q2(3, 3, 2),
    "stokes_2d": lambda: structured_stokes(2, 3, 3),
    "stokes_3d": lambda: structured_stokes(3, 2, 2),
    "scattered_20000": lambda: _scattered(20000),
    "blocks_of_two_1": lambda: _blocks_of_two(1),
    "blocks_of_two_333": lambda: _blocks_of_two(333),
}


def _results(prob, env, nan=False):
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
        ctx.set_params(omega=0.9, smoother="ilu", gmressize=6, tol=1e-30, globaltol=1e-300,
                       maxiter=5)
        out = []
        x, y, h = ctx.vec(), ctx.vec(), ctx.vec()
        for level, lv in enumerate(prob.levels):
            rng = np.random.default_rng(level)
            rhs = rng.standard_normal(lv.ndof)
            if nan:
                rhs[lv.ndof // 3] = np.nan
                rhs[lv.ndof // 2] = np.frombuffer(b"\xff" * 8)[0]  # the kernel's own mark
            ctx.upload(level, x, rng.standard_normal(lv.ndof))
            ctx.upload(level, y, rhs)
            ctx.smooth(level, 2, x, y, h)
            out += [ctx.download(level, x), ctx.download(level, h)]
        fine = prob.nlevels - 1
        ctx.upload(fine, y, prob.rhs)
        if not nan:
            for precision in (GB_FP64, GB_FP32):
                ctx.fgmres(x, y, precision, check=False)
                out.append(ctx.download(fine, x))
        return out


@pytest.mark.parametrize("name", sorted(CASES))
def test_cluster_substitution_equals_level_launches(name):
    prob = CASES[name]()
    for a, b in zip(_results(prob, {}), _results(prob, {"GB_ILU_CTA_ROWS": "0"})):
        assert np.array_equal(a, b)


def test_cluster_substitution_passes_nan_on():
    prob = _diffusion(2, 2, 3)
    for a, b in zip(_results(prob, {}, nan=True),
                    _results(prob, {"GB_ILU_CTA_ROWS": "0"}, nan=True)):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)])
