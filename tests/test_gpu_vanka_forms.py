"""Vanka patches of more than 32 unknowns on either side of the rule that gives a
patch a CTA (few patches) or a warp (many): the patches of a 5^3 node mesh once, and
the same patches repeated past the rule's largest count, whose average is the same.

Tolerance: both sum the same products of a patch's inverse (M of them) in another
order and average up to 8 patches' values, repeated k times; one rounding per
addition, relative to the sums of absolute values: (2 M + 8 k + 8) roundings."""
import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64
from gascoignelib_b200.problem import Level, Problem

pytestmark = pytest.mark.gpu


def _problem(B, repeat):
    """27-point block matrix on 5^3 nodes, the 8 patches of 3^3 nodes `repeat` times."""
    N = 5
    n = N ** 3
    g = np.arange(n).reshape(N, N, N)
    c = np.stack(np.unravel_index(np.arange(n), (N, N, N)), axis=1)
    near = (np.abs(c[:, None, :] - c[None, :, :]) <= 1).all(axis=2)
    row, col = np.nonzero(near)
    ptr = np.concatenate([[0], np.cumsum(near.sum(axis=1))]).astype(np.int64)
    diag = np.flatnonzero(row == col).astype(np.int64)
    rng = np.random.default_rng(B)
    val = rng.uniform(-1.0, 1.0, (col.size, B, B))
    val[diag] += 30.0 * B * np.eye(B)
    patches = np.array([g[2 * k:2 * k + 3, 2 * j:2 * j + 3, 2 * i:2 * i + 3].ravel()
                        for k in range(2) for j in range(2) for i in range(2)], dtype=np.int64)
    level = Level(n=n, B=B, rowptr=ptr, col=col.astype(np.int64), diag=diag, val=val.ravel(),
                  dirichlet=np.array([], dtype=np.int64))
    level.patches = np.tile(patches, (repeat, 1))
    return Problem(dim=3, levels=[level], transfers=[], rhs=rng.standard_normal(n * B),
                   info={"smoother": "vanka"})


@pytest.mark.parametrize("B,repeat", [(2, 125), (2, 126), (3, 250), (3, 251), (4, 375), (4, 376),
                                      (4, 625), (4, 626)])
def test_repeated_patches(ctx, B, repeat):
    sweeps = []
    for k in (1, repeat):
        P = _problem(B, k)
        ctx.load_problem(P)
        ctx.set_params(omega=0.7, smoother="vanka", iterexact=2)
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(0, y, P.rhs)
        for precision in (GB_FP64, GB_FP32):
            ctx.zero(0, x)
            ctx.precondition(x, y, precision)
            sweeps.append(ctx.download(0, x))
        if k == 1:
            M = 27 * B
            inv = np.abs(ctx.vanka_inverse(0, 8, M))
            size = np.einsum("pji,pj->pi", inv, np.abs(P.rhs.reshape(-1, B))[
                P.levels[0].patches].reshape(8, M)).max()
        ctx.free(x)
        ctx.free(y)
    roundings = 2 * M + 8 * repeat + 8
    # two sweeps: the second starts from a residual with the first's difference,
    # which a patch solve passes on with a factor below 2 here (dominant diagonal)
    for one, many, unit in ((sweeps[0], sweeps[2], 1.2e-16), (sweeps[1], sweeps[3], 6e-8)):
        assert np.abs(many).max() > 0.0
        assert np.abs(one - many).max() <= 4 * roundings * unit * size
