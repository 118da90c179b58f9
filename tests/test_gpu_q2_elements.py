"""The Q2 element kernels (matrices on the FP64 matrix unit, matrix-free
residuals) on distorted meshes with a coefficient per element against the
oracle's restatement: one element, fewer than a block's eight, odd counts, 2D
and 3D, with and without convection (without, only the upper tiles are formed).

Tolerance: an entry is a sum of 27 * 4 products of factors with about ten
roundings each, in two different orders: about 120 units of 1.1e-16 on each
side, times the sum of the products' sizes over the largest entry (below 8 on
these meshes): 2e-13 of the largest entry."""
import numpy as np
import pytest

from gascoignelib_b200.problem import Problem, q2_meshes, structured_q2
from oracle.assembly import assemble, q2_element_matrices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("convection", [False, True])
@pytest.mark.parametrize("dim,coarse,refine", [(2, 1, 1), (2, 3, 1), (2, 5, 2), (3, 1, 1),
                                               (3, 3, 1), (3, 2, 2)])
def test_q2_elements_on_distorted_meshes(ctx, dim, coarse, refine, convection):
    P = structured_q2(dim, coarse, refine)
    rng = np.random.default_rng(dim * 100 + coarse)
    fl = P.nlevels - 1
    lv = P.finest
    el = q2_meshes(P)[fl][0]
    n1 = round(lv.n ** (1.0 / dim))
    coord = lv.coord + rng.uniform(-0.15, 0.15, size=lv.coord.shape) / n1
    kappa = np.exp(rng.normal(size=el.shape[0]))
    beta = (1.0, -0.5, 0.25)[:dim] if convection else None
    ctx.load_problem(Problem(dim=dim, levels=[lv], transfers=[], rhs=P.rhs))
    ctx.set_mesh(0, dim, el, coord, None, degree=2)
    ctx.assemble(0, kappa, beta)
    E = q2_element_matrices(dim, coord[el], kappa, beta if convection else (0.0,) * dim)
    want = assemble(lv.n, lv.rowptr, lv.col, el, E, lv.dirichlet)
    got = ctx.level_values(0, lv.val.size)
    assert np.abs(got - want).max() <= 2e-13 * np.abs(want).max()
    x, y = ctx.vec(), ctx.vec()
    u = rng.standard_normal(lv.n)
    ctx.upload(0, x, u)
    ctx.zero(0, y)
    ctx.form(0, y, x)
    f = np.zeros(lv.n)
    np.add.at(f, el, np.einsum("cab,cb->ca", E, u[el]))
    # a sum of 27 entries times values of size 3 more
    assert np.abs(ctx.download(0, y) - f).max() <= 27 * 3 * 2e-13 * np.abs(E).max()
    ctx.free(x)
    ctx.free(y)
