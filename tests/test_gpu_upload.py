"""gb_vec_upload returns when the source has been read: a caller may change it at
once, whether it is pageable (the call does not wait for the device then) or
pinned, from a few values to more than the driver stages in one piece."""
import numpy as np
import pytest
import torch

from gascoignelib_b200.problem import structured_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("dim,coarse,refine", [(2, 2, 1), (2, 2, 5), (3, 1, 6)])
def test_source_may_change_after_upload(ctx, dim, coarse, refine, pinned):
    P = structured_problem(dim, coarse, refine)
    ctx.load_problem(P)
    level, n = P.nlevels - 1, P.finest.n
    src = (torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() if pinned
           else np.empty(n))
    v = ctx.vec()
    for k in range(30):
        src[:] = np.arange(n) + k
        ctx.upload(level, v, src)
        src[:] = -1.0
        assert np.array_equal(ctx.download(level, v), np.arange(n) + float(k))
    ctx.free(v)
