"""Chains whose elements form no long run of one hard operation -- alternating booleans, blends of several
widths, short runs between them, offsets -- are culled by the stretch: kinds against the oracle, accelerated
queries against the whole chain bit for bit, at the edges of a warp's 32 elements and of the run lengths."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _part(X, rng):
    c = rng.uniform(0.05, 0.95, 3)
    k = int(rng.integers(5))
    if k == 0:
        return X.sphere(float(rng.uniform(0.03, 0.12)), c)
    if k == 1:
        return X.box(rng.uniform(0.02, 0.1, 3), c)
    if k == 2:
        return X.capsule(c, c + rng.uniform(-0.1, 0.1, 3), 0.02)
    if k == 3:
        return X.torus(0.06, 0.02, "xyz"[int(rng.integers(3))], c)
    return X.rotate(X.cylinder(0.03, 0.12, center=tuple(c)), "x", float(rng.uniform(0, 90)), about=tuple(c))


def _chain(X, rng, pattern, count):
    t = X.sphere(0.3, (0.5, 0.5, 0.5))
    ops, widths = {"alternate": ("us", (0.0,)), "blends": ("u", (0.01, 0.05)), "cuts": ("us", (0.0, 0.02)),
                   "mixed": ("uusi", (0.0, 0.0, 0.03)), "short_runs": (None, (0.0,)), "wide": ("us", (0.4,))}[pattern]
    i = 0
    while i < count:
        length = 1 if ops else int(rng.integers(1, 12))
        op = ops[int(rng.integers(len(ops)))] if ops else "us"[int(rng.integers(2))]
        if pattern == "alternate":
            op = "us"[i % 2]
        for _ in range(min(length, count - i)):
            k = float(rng.choice(widths))
            p = X.sphere(0.9, rng.uniform(0.3, 0.7, 3)) if op == "i" else _part(X, rng)
            t = {"u": X.union, "s": X.subtract, "i": X.intersect}[op](t, p, k=k)
            i += 1
        if rng.random() < 0.03:
            t = X.offset(t, float(rng.uniform(-2e-3, 2e-3)))
    return t


@pytest.mark.parametrize("pattern", ["alternate", "blends", "cuts", "mixed", "short_runs", "wide"])
@pytest.mark.parametrize("count,n,block", [(4, (40, 40, 40), 8), (31, (64, 50, 41), 8), (33, (130, 60, 40), 4),
                                           (96, (64, 64, 64), 16), (350, (140, 70, 66), 8)])
def test_stretches(pattern, count, n, block):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count)
    comp = X.compile_recipe(_chain(X, rng, pattern, count))
    assert comp.chain is not None
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fb = B.FieldBuilder(comp, meta)
    f = fb.build()
    kind, cma = oracle.classify_program(comp.prims, comp.program, meta)
    assert np.array_equal(f.kind.cpu().numpy(), kind)
    # float32 corner values: 2e-7 a blend of them, of values up to the grid's size
    assert np.abs(fb.cma.cpu().numpy() - cma).max() <= 1e-5 * meta.pitch + 1e-6 * np.abs(cma).max() + 2e-7 * count
    plain, fast = Q.RecipeQueries(comp), Q.RecipeQueries(comp, builder=fb)
    pts = ((rng.uniform(-0.05, 1.05, (45000, 3)) * np.array(n)) / max(n)).astype(np.float32)
    pts = torch.from_numpy(pts).cuda()
    for m in (1500, 45000):
        v0, g0 = plain.values_and_gradients(pts[:m], h=meta.pitch)
        v1, g1 = fast.values_and_gradients(pts[:m], h=meta.pitch)
        assert torch.equal(v0, v1) and torch.equal(g0, g1), m
        assert torch.equal(plain.values(pts[:m]), fast.values(pts[:m])), m
