"""Classification by bricks of blocks equals the float64 oracle for every superblock shape (1 to 512
blocks, ragged grids) and for lists that are a warp's subset as they are, that are culled to its brick, and
that are too long for one."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _recipe(X, rng, count, size, extras):
    parts = []
    for k in range(count):
        c = rng.uniform(0.1, 0.9, 3) * size
        parts.append((X.sphere(float(rng.uniform(0.02, 0.06)), c), X.box(rng.uniform(0.02, 0.06, 3), c),
                      X.capsule(c, c + rng.uniform(-0.08, 0.08, 3), 0.015), X.torus(0.05, 0.015, "xyz"[k % 3], c))[k % 4])
    t = X.subtract_all(X.union_all(parts), [X.capsule(rng.uniform(0, 1, 3) * size, rng.uniform(0, 1, 3) * size, 0.01)
                                            for _ in range(count // 8)])
    if extras:  # elements that step one at a time, and a run behind them
        t = X.intersect(X.offset(X.union(t, X.cylinder(0.05, 0.4, center=tuple(0.5 * size)), k=0.03), 0.002),
                        X.sphere(0.8, tuple(0.5 * size)))
        t = X.subtract_all(t, [X.sphere(0.04, rng.uniform(0.2, 0.8, 3) * size) for _ in range(5)])
    return t


@pytest.mark.parametrize("n,block,count,extras", [
    ((130, 70, 41), 4, 12, True), ((130, 70, 41), 4, 300, False), ((129, 40, 40), 4, 1500, True),
    ((150, 90, 67), 8, 200, True), ((140, 64, 64), 8, 1500, False), ((140, 64, 50), 16, 60, True),
    ((64, 50, 33), 4, 40, False), ((60, 40, 37), 4, 700, True), ((100, 50, 41), 8, 90, True), ((80, 64, 48), 16, 30, False)])
def test_bricks_equal_the_oracle(n, block, count, extras):
    import field_b200.build as B
    import field_b200.expr as X
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count + block)
    size = np.array(n) / max(n)
    comp = X.compile_recipe(_recipe(X, rng, count, size, extras))
    assert comp.chain is not None
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fb = B.FieldBuilder(comp, meta)
    f = fb.build()
    kind, cma = oracle.classify_program(comp.prims, comp.program, meta)
    assert np.array_equal(f.kind.cpu().numpy(), kind)
    # float32 evaluation in block-local coordinates: the leaves' own bound
    assert np.abs(fb.cma.cpu().numpy() - cma).max() <= 1e-5 * meta.pitch + 1e-6 * np.abs(cma).max()
    ids = rng.permutation(np.where(kind == 0)[0])[:300]
    slot = np.searchsorted(f.active[:f.n_active].cpu().numpy(), ids)
    want = oracle.tiles_program(comp.prims, comp.program, meta, ids.astype(np.int32)).reshape(len(ids), -1)
    got = f.tiles[:f.n_active].cpu().numpy()[slot]
    near = np.abs(want) <= 3 * meta.pitch
    assert np.abs(got - want)[near].max() <= 1e-5 * meta.pitch
    assert np.array_equal(got >= 0, want >= 0)
