"""Accelerated queries of primitives whose frames are far larger than the grid (their float32 values carry
the rounding of those frames) equal the whole chain's bit for bit: surfaces that nearly coincide, steps and
point spacings below that rounding, steep half-spaces, and fields built with a raised guard band."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


P0 = np.array([0.51, 0.53, 0.47])


def _directions(rng, n, spread):
    d = np.array([0.8, 0.5, 0.33]) + rng.normal(size=(n, 3)) * spread
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _spheres(X, rng):  # all through P0, radii of hundreds: float32 values there are off by up to 4e-5
    return X.union_all([X.sphere(float(r), P0 + (r + rng.uniform(-2e-5, 2e-5)) * d)
                        for d, r in zip(_directions(rng, 24, 0.2), rng.uniform(100, 600, 24))])


def _tori(X, rng):
    parts = [X.torus(float(r), float(r) / 2, "xyz"[k % 3], P0 + (1.5 * r + rng.uniform(-2e-5, 2e-5)) * np.eye(3)[(k + 1) % 3])
             for k, r in enumerate(rng.uniform(100, 400, 18))]
    return X.union(X.union_all(parts), X.box((0.1, 0.1, 0.1), (0.3, 0.3, 0.3)), k=0.01)


def _boxes(X, rng):
    parts = []
    for k, e in enumerate(rng.uniform(200, 500, 16)):
        axis = np.eye(3)[k % 3]
        parts.append(X.rotate(X.box((float(e),) * 3, P0 + (e + rng.uniform(-2e-5, 2e-5)) * axis), "xyz"[(k + 1) % 3],
                              float(rng.uniform(-5, 5)), about=tuple(P0)))
    return X.subtract_all(X.sphere(0.45, (0.5, 0.5, 0.5)), parts)


def _halfspaces(X, rng):
    d = np.array([0.6, 0.64, 0.48])
    parts = [{"op": "halfspace", "normal": [float(v) for v in 40.0 * d],
              "offset": float((0.8 + rng.uniform(-1e-6, 1e-6)) / 40.0)} for _ in range(16)]
    return X.intersect(X.union_all(parts), X.sphere(0.6, (0.5, 0.5, 0.5)))


@pytest.mark.parametrize("make", [_spheres, _tori, _boxes, _halfspaces])
@pytest.mark.parametrize("guard", [None, 1e-3])
def test_large_frames_equal_the_whole_chain(make, guard):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(11)
    comp = X.compile_recipe(make(X, rng))
    assert comp.chain is not None
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / 64, 64, 64, 64, 8)
    fb = B.FieldBuilder(comp, meta, guard=guard)
    fb.classify()
    plain, fast = Q.RecipeQueries(comp), Q.RecipeQueries(comp, builder=fb)
    # clusters of close points (the sorted path's groups span a cluster), some around the near-coincident surfaces
    at = rng.uniform(0.1, 0.9, (500, 1, 3))
    at[::2, 0] = P0 + rng.normal(size=(250, 3)) * 10.0 ** rng.uniform(-6, -3, (250, 1))
    pts = (at + rng.uniform(-1, 1, (500, 100, 3)) * 10.0 ** rng.uniform(-7, -4, (500, 1, 1))).reshape(-1, 3)
    pts = torch.from_numpy(pts.astype(np.float32)).cuda()
    for m in (4000, 50000):
        for h in (1e-7, 1e-6, 1e-5, 1.0 / 64):
            v0, g0 = plain.values_and_gradients(pts[:m], h=h)
            v1, g1 = fast.values_and_gradients(pts[:m], h=h)
            assert torch.equal(v0, v1) and torch.equal(g0, g1), (m, h)
        assert torch.equal(fast.values(pts[:m]), plain.values(pts[:m])), m
