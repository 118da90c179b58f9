"""Products and residuals with rows of more than 32 entries, on either side of
the size rules (a slice shared by four warps up to 32,768 rows, one thread per
row above), against scipy: row lengths that leave some of the four warps
without columns or end inside a group of four, one row, a last slice that is
not full, column patterns, 16-bit offsets and plain columns.

Tolerance: sums of at most 131 products in two orders, 2 * 131 * 1.1e-16 of the
sum of their sizes."""
import numpy as np
import pytest
import scipy.sparse as sp

from gascoignelib_b200.problem import Level, Problem

pytestmark = pytest.mark.gpu


def _matrix(n, width, kind, rng):
    """Rows of 1 to `width` entries (always the diagonal): "pattern", the same
    offsets everywhere; "near", random columns within 2^15; "far", anywhere."""
    if kind == "pattern":
        offs = np.arange(width) - width // 2
        a = sp.diags([rng.standard_normal(n) for _ in offs], offs, shape=(n, n), format="csr")
    else:
        reach = min(n, 30000 if kind == "near" else n)
        rows = []
        for i in range(n):
            lo = max(0, min(i - reach // 2, n - reach))
            k = int(rng.integers(1, width + 1)) if i % 7 else width
            cols = np.unique(np.append(lo + rng.integers(0, reach, size=min(k, n) - 1), i))
            rows.append(cols)
        ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])])
        col = np.concatenate(rows)
        a = sp.csr_matrix((rng.standard_normal(col.size), col, ptr), shape=(n, n))
    a = (a + sp.identity(n) * 3.0).tocsr()
    a.sort_indices()
    return a


@pytest.mark.parametrize("n,width,kind", [
    (1, 1, "near"), (33, 33, "pattern"), (97, 35, "near"), (1000, 37, "pattern"),
    (1025, 131, "near"), (2048, 49, "far"), (32768, 40, "pattern"), (32769, 40, "pattern"),
    (40000, 70, "near"), (70001, 60, "far")])
def test_products_with_long_rows(ctx, n, width, kind):
    rng = np.random.default_rng(n)
    a = _matrix(n, width, kind, rng)
    ptr, col = a.indptr.astype(np.int64), a.indices.astype(np.int64)
    ri = np.repeat(np.arange(n), np.diff(ptr))
    lv = Level(n=n, B=1, rowptr=ptr, col=col, diag=np.nonzero(ri == col)[0].astype(np.int64),
               val=a.data.copy(), dirichlet=np.array([0], dtype=np.int64))
    ctx.load_problem(Problem(dim=2, levels=[lv], transfers=[], rhs=np.zeros(n)))
    xv, bv = rng.standard_normal(n), rng.standard_normal(n)
    x, y, b = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.upload(0, x, xv)
    ctx.upload(0, b, bv)
    want = a @ xv
    bound = 2 * 131 * 1.1e-16 * (abs(a) @ np.abs(xv) + np.abs(bv))
    ctx.vmulteq(0, y, x)
    assert np.all(np.abs(ctx.download(0, y) - want) <= bound)
    ctx.upload(0, y, bv)
    ctx.vmult(0, y, x, 0.5)
    assert np.all(np.abs(ctx.download(0, y) - (bv + 0.5 * want)) <= bound)
    ctx.residualgmres(0, y, x, b)
    r = bv - want
    r[0] = 0.0  # the Dirichlet row
    assert np.all(np.abs(ctx.download(0, y) - r) <= bound)
    ctx.set_params(omega=0.3)
    ctx.smooth_jacobi(0, 1, x, b, y)
    d = 1.0 / a.diagonal()
    got = ctx.download(0, x)
    assert np.all(np.abs(got - (xv + 0.3 * d * (bv - want)))
                  <= 0.3 * np.abs(d) * bound + 4 * 1.1e-16 * (np.abs(xv) + np.abs(0.3 * d * (bv - want))))
    for v in (x, y, b):
        ctx.free(v)
