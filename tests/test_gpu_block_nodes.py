"""Block transfers and the Vanka average on either side of the rule that gives a
thread one component of a node (small levels) or all of them: 2D meshes just below
and just above 70,000 nodes, block sizes 2 to 4, against numpy.

Matrices are block-diagonal, so that a Vanka patch's solution is the block inverse
times the right-hand side at each of its nodes, whatever the patch.

Tolerance: transfers add at most 9 values with weights that are powers of two (9
roundings); an average adds at most 4 patches' values, each a sum of 4 products with
an inverse that is itself within a few roundings of numpy's (64 roundings)."""
import dataclasses

import numpy as np
import pytest

from gascoignelib_b200.native import GB_FP32, GB_FP64
from gascoignelib_b200.problem import Level, Problem, structured_problem

pytestmark = pytest.mark.gpu

EPS = 1.2e-16


def _problem(B, coarse):
    """The transfers of a mesh of (4 coarse)^2 cells, two levels of B components."""
    S = structured_problem(2, coarse, 2)
    rng = np.random.default_rng(B)
    levels = []
    for lv in S.levels:
        val = rng.uniform(-1.0, 1.0, (lv.n, B, B)) + 4.0 * B * np.eye(B)
        L = Level(n=lv.n, B=B, rowptr=np.arange(lv.n + 1, dtype=np.int64),
                  col=np.arange(lv.n, dtype=np.int64), diag=np.arange(lv.n, dtype=np.int64),
                  val=val.ravel(), dirichlet=np.array([], dtype=np.int64))
        N = int(round(lv.n ** 0.5))
        i = np.arange(0, N - 2, 2)
        corner = (i[:, None] * N + i[None, :]).ravel()
        local = (np.arange(3)[:, None] * N + np.arange(3)[None, :]).ravel()
        L.patches = (corner[:, None] + local[None, :]).astype(np.int64)
        levels.append(L)
    return Problem(dim=2, levels=levels, transfers=S.transfers,
                   rhs=rng.standard_normal(levels[-1].ndof), info={"smoother": "vanka"})


# nodes of the fine level 261^2 and 265^2; of the coarse one 261^2 and 265^2
@pytest.mark.parametrize("B,coarse", [(2, 65), (2, 66), (3, 65), (3, 66), (4, 65), (4, 66),
                                      (3, 130), (3, 132)])
def test_block_transfers(ctx, B, coarse):
    P = _problem(B, coarse)
    ctx.load_problem(P)
    T, (Lc, Lf) = P.transfers[0], P.levels
    rng = np.random.default_rng(7)
    uc, uf = rng.standard_normal((Lc.n, B)), rng.standard_normal((Lf.n, B))
    # the nodal interpolation and its transpose
    up, upabs, down = np.zeros((Lf.n, B)), np.zeros((Lf.n, B)), np.zeros((Lc.n, B))
    downabs = np.zeros((Lc.n, B))
    pairs = [(T.c2f, np.arange(Lc.n), 1.0)]
    pairs += [(T.zweier[:, 0], T.zweier[:, k], 0.5) for k in (1, 2)]
    pairs += [(T.vierer[:, 0], T.vierer[:, k], 0.25) for k in (1, 2, 3, 4)]
    for f, c, w in pairs:
        np.add.at(up, f, w * uc[c])
        np.add.at(upabs, f, w * np.abs(uc[c]))
        np.add.at(down, c, w * uf[f])
        np.add.at(downabs, c, w * np.abs(uf[f]))
    c, f = ctx.vec(), ctx.vec()
    ctx.upload(0, c, uc.ravel())
    ctx.upload(1, f, uf.ravel())
    ctx.prolongate_add(0, f, c)
    assert np.all(np.abs(ctx.download(1, f) - (uf + up).ravel())
                  <= 9 * EPS * (np.abs(uf) + upabs).ravel())
    ctx.upload(1, f, uf.ravel())
    ctx.restrict_zero(0, c, f)
    assert np.all(np.abs(ctx.download(0, c) - down.ravel()) <= 9 * EPS * downabs.ravel())
    ctx.free(c)
    ctx.free(f)


@pytest.mark.parametrize("B,coarse", [(2, 65), (2, 66), (3, 65), (3, 66), (4, 65), (4, 66)])
def test_vanka_average(ctx, B, coarse):
    P = dataclasses.replace(_problem(B, coarse), transfers=[])
    P.levels = P.levels[1:]
    lv = P.levels[0]
    ctx.load_problem(P)
    ctx.set_params(omega=0.7, smoother="vanka", iterexact=1)
    bv = P.rhs.reshape(-1, B)
    inv = np.linalg.inv(lv.val.reshape(-1, B, B))
    want = 0.7 * np.einsum("nij,nj->ni", inv, bv)
    size = np.einsum("nij,nj->ni", np.abs(inv), np.abs(bv))
    x, y = ctx.vec(), ctx.vec()
    ctx.upload(0, y, P.rhs)
    for precision, unit in ((GB_FP64, EPS), (GB_FP32, 6e-8)):
        ctx.zero(0, x)
        ctx.precondition(x, y, precision)
        got = ctx.download(0, x).reshape(-1, B)
        assert np.all(np.abs(got - want) <= 64 * unit * size)
    ctx.free(x)
    ctx.free(y)
