"""Block products and residuals on either side of the size rule that gives a row a
thread or B threads, for every block size and for rows of 9 and of 27 blocks.

Tolerance: a row is a sum of at most 27 * 4 products in FP64, in two orders:
2 * 108 * 1.2e-16 of the sum of their sizes."""
import numpy as np
import pytest

from gascoignelib_b200.problem import Level, Problem

pytestmark = pytest.mark.gpu


def _level(dim, N, B):
    """The 3^dim-point block matrix of an N^dim grid."""
    n = N ** dim
    c = np.stack(np.unravel_index(np.arange(n), (N,) * dim), axis=1)
    offs = np.stack(np.meshgrid(*[[-1, 0, 1]] * dim, indexing="ij"), axis=-1).reshape(-1, dim)
    q = c[:, None, :] + offs
    keep = ((q >= 0) & (q < N)).all(axis=2)
    cols = np.ravel_multi_index(np.moveaxis(np.clip(q, 0, N - 1), 2, 0), (N,) * dim)
    ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int64)
    diag = ptr[:-1] + keep[:, :len(offs) // 2].sum(axis=1)
    val = np.random.default_rng(N).uniform(-1.0, 1.0, (int(ptr[-1]), B, B))
    val[diag] += 30.0 * np.eye(B)
    return Level(n=n, B=B, rowptr=ptr, col=cols[keep].astype(np.int64), diag=diag, val=val.ravel(),
                 dirichlet=np.array([], dtype=np.int64))


@pytest.mark.parametrize("dim,N,B", [(2, 219, 2), (2, 220, 2), (2, 282, 3), (2, 283, 3),
                                     (2, 181, 4), (2, 182, 4), (3, 41, 2), (3, 42, 2),
                                     (3, 46, 3), (3, 47, 3)])
def test_products_and_residuals(ctx, dim, N, B):
    lv = _level(dim, N, B)
    ctx.load_problem(Problem(dim=dim, levels=[lv], transfers=[], rhs=np.zeros(lv.ndof)))
    rng = np.random.default_rng(B)
    xv, bv = rng.standard_normal(lv.ndof), rng.standard_normal(lv.ndof)

    def product(val, x):
        parts = np.einsum("erc,ec->er", val.reshape(-1, B, B), x.reshape(-1, B)[lv.col])
        return np.add.reduceat(parts, lv.rowptr[:-1], axis=0).ravel()

    want = product(lv.val, xv)
    bound = 2 * 108 * 1.2e-16 * (product(np.abs(lv.val), np.abs(xv)) + np.abs(bv))
    x, y, b = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.upload(0, x, xv)
    ctx.upload(0, b, bv)
    ctx.vmulteq(0, y, x)
    assert np.all(np.abs(ctx.download(0, y) - want) <= bound)
    ctx.matrix_residual(0, y, x, b)
    assert np.all(np.abs(ctx.download(0, y) - (bv - want)) <= bound)
    for v in (x, y, b):
        ctx.free(v)
