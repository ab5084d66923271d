"""A boolean of negative blend width is the hard one, in the culling as in the evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(X, k):
    rng = np.random.default_rng(3)
    t = X.sphere(0.3, (0.4, 0.4, 0.4))
    for i in range(60):
        c = tuple(rng.uniform(0.1, 0.9, 3))
        part = X.sphere(0.1, c) if i % 2 else X.box((0.08, 0.05, 0.07), c)
        t = X.subtract(t, part, k=k) if i % 5 == 4 else X.union(t, part, k=k)
    return X.intersect(t, X.sphere(0.55, (0.5, 0.5, 0.5)), k=k)


@pytest.mark.parametrize("n,block", [((64, 64, 64), 8), ((70, 50, 41), 4), ((150, 40, 40), 8), ((64, 64, 64), 16)])
def test_negative_width_equals_hard(n, block):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fields, values = [], []
    pts = torch.rand((3000, 3), generator=torch.Generator().manual_seed(1)).cuda()
    for k in (0.0, -0.15):
        comp = X.compile_recipe(_recipe(X, k))
        assert comp.chain is not None
        fb = B.FieldBuilder(comp, meta)
        fields.append(fb.build())
        values.append(Q.RecipeQueries(comp, builder=fb).values_and_gradients(pts, h=meta.pitch))
    a, b = fields
    assert torch.equal(a.kind, b.kind) and a.n_active == b.n_active
    assert torch.equal(a.tiles[:a.n_active], b.tiles[:b.n_active]) and torch.equal(a.corner_min_abs, b.corner_min_abs)
    assert torch.equal(values[0][0], values[1][0]) and torch.equal(values[0][1], values[1][1])
