"""gb_vec_upload from sources that change at once, around the size up to which it
goes through the context's own pinned buffer, while kernels and earlier uploads are
still under way: several uploads in a row reuse that buffer."""
import numpy as np
import pytest

from gascoignelib_b200.native import Context
from gascoignelib_b200.problem import structured_problem

pytestmark = pytest.mark.gpu


# 33^2 nodes; 32,761 (below 256 KB) and 33,489 nodes (above); one of the two levels
@pytest.mark.parametrize("coarse,refine", [(2, 4), (45, 2), (91, 1)])
def test_uploads_in_a_row(coarse, refine):
    P = structured_problem(2, coarse, refine)
    with Context(0) as ctx:
        ctx.load_problem(P)
        fine = P.nlevels - 1
        n = P.finest.n
        vecs = [ctx.vec() for _ in range(6)]
        x, y = ctx.vec(), ctx.vec()
        ctx.upload(fine, y, np.random.default_rng(0).standard_normal(n))
        src = np.empty(n)
        for k in range(5):
            for _ in range(3):
                ctx.precondition(x, y)  # the stream is busy
            for i, v in enumerate(vecs):
                src[:] = np.arange(n) + 100 * k + i
                ctx.upload(fine, v, src)
                src[:] = -1.0
            for i, v in enumerate(vecs):
                assert np.array_equal(ctx.download(fine, v), np.arange(n) + 100.0 * k + i)
