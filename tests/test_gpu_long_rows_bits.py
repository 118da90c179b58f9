"""Rows of more than 32 entries on small levels, whose slices four warps share: the
sums run in the entries' order, so the product in FP64 is, bit for bit, the chain
acc = fma(a_j, x_j, acc), here in exact rational arithmetic rounded once per step.
Row lengths that end inside a warp's columns and after whole turns, one row, a last
slice that is not full, column patterns, 16-bit offsets and plain columns."""
from fractions import Fraction

import numpy as np
import pytest
import scipy.sparse as sp

from gascoignelib_b200.problem import Level, Problem

pytestmark = pytest.mark.gpu


def _chain(row_cols, row_vals, x, start=0.0, sign=1.0):
    acc = start
    for c, v in zip(row_cols, row_vals):
        acc = float(Fraction(sign * v) * Fraction(x[c]) + Fraction(acc))
    return acc


@pytest.mark.parametrize("n,width,kind", [(1, 1, "near"), (40, 33, "near"), (129, 48, "pattern"),
                                          (100, 64, "near"), (161, 65, "far"), (200, 125, "near"),
                                          (150, 131, "pattern")])
def test_sums_in_the_entries_order(ctx, n, width, kind):
    rng = np.random.default_rng(n)
    if kind == "pattern":
        offs = np.arange(width) - width // 2
        a = sp.diags([rng.standard_normal(n) for _ in offs], offs, shape=(n, n), format="csr")
    else:
        rows = [np.unique(np.append(rng.integers(0, n, size=width if i % 7 == 0 else
                                                 int(rng.integers(1, width + 1))), i))
                for i in range(n)]
        ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])])
        col = np.concatenate(rows)
        a = sp.csr_matrix((rng.standard_normal(col.size), col, ptr), shape=(n, n))
    a = (a + 3.0 * sp.identity(n)).tocsr()
    a.sort_indices()
    ptr, col, val = a.indptr.astype(np.int64), a.indices.astype(np.int64), a.data
    ri = np.repeat(np.arange(n), np.diff(ptr))
    lv = Level(n=n, B=1, rowptr=ptr, col=col, diag=np.nonzero(ri == col)[0].astype(np.int64),
               val=val.copy(), dirichlet=np.array([], dtype=np.int64))
    ctx.load_problem(Problem(dim=2, levels=[lv], transfers=[], rhs=np.zeros(n)))
    xv, bv = rng.standard_normal(n), rng.standard_normal(n)
    x, y, b = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.upload(0, x, xv)
    ctx.upload(0, b, bv)
    row = [(col[ptr[i]:ptr[i + 1]], val[ptr[i]:ptr[i + 1]]) for i in range(n)]
    ctx.vmulteq(0, y, x)
    assert np.array_equal(ctx.download(0, y), [_chain(*r, xv) for r in row])
    ctx.residualgmres(0, y, x, b)
    assert np.array_equal(ctx.download(0, y),
                          [_chain(*r, xv, bv[i], -1.0) for i, r in enumerate(row)])
    for v in (x, y, b):
        ctx.free(v)
