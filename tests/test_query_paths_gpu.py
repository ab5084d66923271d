"""Accelerated point queries equal the whole chain's, bit for bit, on every path: a warp per point (few
points), points sorted by cell, and the variants and points that leave a superblock's ball."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(X, rng, n, extras):
    size = np.array(n) / max(n)
    parts = []
    for k in range(40):
        c = rng.uniform(0.1, 0.9, 3) * size
        parts.append((X.sphere(0.05, c), X.box((0.04, 0.06, 0.03), c), X.capsule(c, c + 0.1, 0.02),
                      X.torus(0.07, 0.02, "xyz"[k % 3], c))[k % 4])
    t = X.subtract_all(X.union_all(parts), [X.capsule(rng.uniform(0, 1, 3) * size, rng.uniform(0, 1, 3) * size, 0.01)
                                            for _ in range(6)])
    if extras:  # smooth booleans, an offset, kinds off the common four, a turned frame
        t = X.union(t, X.cylinder(0.05, 0.4, center=tuple(0.5 * size)), k=0.05)
        t = X.offset(t, 0.004)
        t = X.intersect(t, X.halfspace((0.0, 0.6, 0.8), 0.7), k=0.02)
        t = X.union(t, X.rotate(X.cone(0.06, 0.02, 0.2, center=tuple(0.3 * size)), "x", 33.0), k=0.0)
    return t


@pytest.mark.parametrize("n,block,extras", [((64, 48, 33), 8, True), ((130, 70, 51), 4, False), ((90, 200, 61), 16, True),
                                            ((7, 9, 5), 4, False)])
def test_paths_equal_the_whole_chain(n, block, extras):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(block)
    comp = X.compile_recipe(_recipe(X, rng, n, extras))
    assert comp.chain is not None
    pitch = 1.0 / max(n)
    meta = GridMeta(0.0, 0.0, 0.0, pitch, *n, block)
    fb = B.FieldBuilder(comp, meta)
    fb.classify()
    plain, fast = Q.RecipeQueries(comp), Q.RecipeQueries(comp, builder=fb)
    size = torch.tensor(n, dtype=torch.float64) * pitch
    gen = torch.Generator().manual_seed(block)
    pts = (torch.rand((50000, 3), generator=gen, dtype=torch.float64) * 1.1 - 0.05) * size
    pts[:2000] = torch.round(pts[:2000] / pitch) * pitch  # on vertices: block, superblock and grid faces
    pts = pts.float()
    pts[7], pts[8] = float("nan"), float("inf")
    pts[9] = torch.tensor([50.0, -30.0, 0.5])
    pts = pts.cuda()
    same = lambda a, b: torch.equal(a.nan_to_num(nan=1e30), b.nan_to_num(nan=1e30))
    # around the switch from a warp per point to sorted points, warps that are not full
    for m, h in [(1, pitch), (31, 0.05), (40960, pitch), (40961, pitch), (50000, 1e-4), (50000, 0.3), (500, 3.0)]:
        v0, g0 = plain.values_and_gradients(pts[:m], h=h)
        v1, g1 = fast.values_and_gradients(pts[:m], h=h)
        assert same(v0, v1) and same(g0, g1), (m, h)
        assert same(fast.values(pts[:m]), v0), m
        g2 = torch.empty_like(g0)
        fast._run(pts[:m].contiguous(), None, g2, h=h)
        assert same(g2, g0), (m, h)
