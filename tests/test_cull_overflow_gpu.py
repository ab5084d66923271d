"""More parts in one coarse region than its list holds, followed by elements that step one at a time: the region
falls back to the whole chain, and nothing that comes later is decided by bounds from before the overflow."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

N, BLOCK, PITCH = (8192, 8192, 32), 16, 1.0 / 64  # 128 x 128 coarse regions: 1024 list entries each
CORNER = np.array([4096, 2048, 0])  # the crowded region's first voxel


def _crowd(X, rng, count):
    return [X.sphere(float(rng.uniform(0.7, 1.5)) * PITCH, (CORNER + rng.uniform(0, 1, 3) * (64, 64, 32)) * PITCH)
            for _ in range(count)]


def _recipe(X, rng, kind, count):
    parts = _crowd(X, rng, count)
    mid = (CORNER + (32, 32, 16)) * PITCH
    if kind == "union":
        t = X.union(X.union_all([X.sphere(0.5, (1.0, 1.0, 0.2))] + parts), X.sphere(3 * PITCH, mid), k=0.05)
        return X.offset(t, 0.002)
    t = X.subtract_all(X.box((100.0, 100.0, 10.0), (64.0, 64.0, 0.2)), parts)
    t = X.subtract(t, X.sphere(3 * PITCH, mid), k=0.05)
    return t if kind == "subtract" else X.intersect(t, X.sphere(0.6, mid), k=0.02)


@pytest.mark.parametrize("kind", ["union", "subtract", "intersect"])
@pytest.mark.parametrize("count", [1000, 1100, 1500])
def test_crowded_region(kind, count):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count)
    comp = X.compile_recipe(_recipe(X, rng, kind, count))
    assert comp.chain is not None
    meta = GridMeta(0.0, 0.0, 0.0, PITCH, *N, BLOCK)
    fb = B.FieldBuilder(comp, meta)
    fb.classify()
    # the crowded region as a grid of its own (every coordinate a multiple of a power of two: the same bits)
    sub = GridMeta(*(CORNER * PITCH), PITCH, 64, 64, 32, BLOCK)
    want, cma = oracle.classify_program(comp.prims, comp.program, sub)
    at = CORNER // BLOCK
    grid = (meta.n_bx, meta.n_by, meta.n_bz)
    here = lambda a: a.reshape(grid)[at[0]:at[0] + 4, at[1]:at[1] + 4, at[2]:at[2] + 2].cpu().numpy().reshape(-1)
    assert np.array_equal(here(fb.kind), want)
    assert np.abs(here(fb.cma) - cma).max() <= 1e-5 * PITCH + 1e-6 * 128
    pts = torch.from_numpy(((CORNER + rng.uniform(0, 1, (4000, 3)) * (64, 64, 32)) * PITCH).astype(np.float32)).cuda()
    v0, g0 = Q.RecipeQueries(comp).values_and_gradients(pts, h=PITCH)
    v1, g1 = Q.RecipeQueries(comp, builder=fb).values_and_gradients(pts, h=PITCH)
    assert torch.equal(v0, v1) and torch.equal(g0, g1)
