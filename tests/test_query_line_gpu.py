"""The line between the two accelerated query paths, for values and for gradients: on both sides of it the
values are the whole chain's, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,block", [((64, 64, 64), 8), ((40, 33, 9), 4), ((200, 150, 170), 8), ((500, 400, 420), 16)])
def test_both_sides_of_the_line(n, block):
    import torch
    import field_b200._lib as L
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(block)
    t = X.union_all([X.sphere(0.06, rng.uniform(0.1, 0.8, 3)) if k % 2 else X.box((0.05, 0.04, 0.06), rng.uniform(0.1, 0.8, 3))
                     for k in range(60)])
    comp = X.compile_recipe(t)
    fb = B.FieldBuilder(comp, GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block))
    fb.classify()
    plain, fast = Q.RecipeQueries(comp), Q.RecipeQueries(comp, builder=fb)
    dims = np.array([*n, block], np.int32)
    needs = lambda m, grad: L.lib().fb_query_scratch_bytes(dims.ctypes.data, m, grad) > 0
    pts = torch.rand((40962, 3), generator=torch.Generator().manual_seed(block)).cuda()
    for grad in (0, 1):
        lo, hi = 1, 40961  # the last count without scratch
        assert not needs(lo, grad) and needs(hi, grad)
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (lo, mid) if needs(mid, grad) else (mid, hi)
        assert (lo == 40960) if grad else (15000 < lo <= 40960)
        for m in (lo, lo + 1):
            if grad:
                v0, g0 = plain.values_and_gradients(pts[:m], h=1.0 / max(n))
                v1, g1 = fast.values_and_gradients(pts[:m], h=1.0 / max(n))
                assert torch.equal(v0, v1) and torch.equal(g0, g1), m
            else:
                assert torch.equal(plain.values(pts[:m]), fast.values(pts[:m])), m
