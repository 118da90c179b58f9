"""Block-level kernels on either side of their size rule: the product and the
residual with a thread per row and component (small levels) and per row (above
100,000 rows), and the Vanka sweep of large patches (108 unknowns, one CTA
each), against numpy.

Tolerance: a row is a sum of at most 27 * 4 products in FP64, in two orders:
2 * 108 * 1.1e-16 of the sum of their sizes; the Vanka sweep adds a product with
a 108-column inverse, whose entries' sizes enter the sum."""
import numpy as np
import pytest

from gascoignelib_b200.problem import structured_stokes

pytestmark = pytest.mark.gpu


def _product(lv, x, absolute=False):
    val, xb = lv.val.reshape(-1, lv.B, lv.B), x.reshape(-1, lv.B)
    if absolute:
        val, xb = np.abs(val), np.abs(xb)
    parts = np.einsum("erc,ec->er", val, xb[lv.col])
    return np.add.reduceat(parts, lv.rowptr[:-1], axis=0).ravel()


@pytest.mark.parametrize("dim,coarse,refine", [(2, 2, 1), (2, 3, 3), (3, 2, 2), (3, 3, 2), (2, 5, 6)])
def test_block_products(ctx, dim, coarse, refine):
    P = structured_stokes(dim, coarse, refine)
    ctx.load_problem(P)
    lv, level = P.finest, P.nlevels - 1
    rng = np.random.default_rng(coarse)
    xv, bv = rng.standard_normal(lv.ndof), rng.standard_normal(lv.ndof)
    x, y, b = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.upload(level, x, xv)
    ctx.upload(level, b, bv)
    want = _product(lv, xv)
    bound = 2 * 108 * 1.1e-16 * (_product(lv, xv, True) + np.abs(bv))
    ctx.vmulteq(level, y, x)
    assert np.all(np.abs(ctx.download(level, y) - want) <= bound)
    ctx.upload(level, y, bv)
    ctx.vmult(level, y, x, -2.0)
    assert np.all(np.abs(ctx.download(level, y) - (bv - 2.0 * want)) <= 2 * bound)
    for v in (x, y, b):
        ctx.free(v)


@pytest.mark.parametrize("dim,coarse,refine", [(3, 2, 1), (3, 3, 2), (2, 3, 2)])
def test_vanka_sweep_of_patches(ctx, dim, coarse, refine):
    """One sweep from x = 0 with the filter off: omega times the average over
    its patches of the patch inverses times the right-hand side."""
    P = structured_stokes(dim, coarse, refine)
    lv, level = P.finest, P.nlevels - 1
    lv.pf_mask = 0
    ctx.load_problem(P)
    ctx.set_params(omega=0.7, smoother="vanka")
    npatch, npp = lv.patches.shape
    M = npp * lv.B
    rng = np.random.default_rng(9)
    bv = rng.standard_normal(lv.ndof)
    x, y, h = ctx.vec(), ctx.vec(), ctx.vec()
    ctx.zero(level, x)
    ctx.upload(level, y, bv)
    ctx.smooth(level, 1, x, y, h)
    inv = ctx.vanka_inverse(level, npatch, M)  # [p, j, i]: column j
    rhs = bv.reshape(-1, lv.B)[lv.patches].reshape(npatch, M)
    sol = np.einsum("pji,pj->pi", inv, rhs)
    size = np.einsum("pji,pj->pi", np.abs(inv), np.abs(rhs))
    out, top, cnt = (np.zeros((lv.n, lv.B)) for _ in range(3))
    np.add.at(out, lv.patches, sol.reshape(npatch, npp, lv.B))
    np.add.at(top, lv.patches, size.reshape(npatch, npp, lv.B))
    np.add.at(cnt, lv.patches, 1.0)
    got = ctx.download(level, x).reshape(lv.n, lv.B)
    assert np.all(np.abs(got - 0.7 * out / cnt) <= 2 * (M + 8 + 2) * 1.1e-16 * top / cnt + 1e-300)
    for v in (x, y, h):
        ctx.free(v)
