"""A half-space's value is n . x for a normal of any length: its bounds widen with that length, so culling
(chains) and pruning (general programs) keep what a unit normal's bounds would drop."""
import numpy as np
import pytest

import oracle


def _halfspace(normal, offset):
    return {"op": "halfspace", "normal": [float(v) for v in normal], "offset": float(offset)}


def _recipe(X, length, chain):
    """Half-spaces that fall `length` times as fast as the unit ones that rise against them."""
    d = np.ones(3) / np.sqrt(3.0)
    steep = _halfspace(length * d, 0.8 / length)  # length (d . x - 0.8)
    gentle = _halfspace(-d, -0.9)  # 0.9 - d . x
    if chain:
        return X.intersect(X.union(gentle, steep), X.sphere(0.8, (0.5, 0.5, 0.5)))
    inner = X.union(X.union(gentle, steep), X.subtract(X.sphere(0.1, (0.2, 0.2, 0.2)), X.sphere(0.06, (0.2, 0.2, 0.3))))
    return X.intersect(X.sphere(0.8, (0.5, 0.5, 0.5)), X.union(inner, X.subtract(
        X.box((0.1, 0.1, 0.1), (0.8, 0.2, 0.3)), X.sphere(0.05, (0.8, 0.2, 0.3)))))


@pytest.mark.parametrize("length", [3.0, 1.0, 0.25])
def test_host_bound(length):
    import field_b200.expr as X
    c = X.compile_recipe(_halfspace((0.0, 0.6 * length, 0.8 * length), 0.1))
    assert c.lipschitz()[0] == pytest.approx(length, rel=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("chain", [True, False])
@pytest.mark.parametrize("length", [3.0, 12.0, 0.25])
@pytest.mark.parametrize("n,block", [((64, 64, 64), 8), ((61, 40, 70), 4), ((64, 50, 48), 16)])
def test_fields_with_any_normal(n, block, length, chain):
    import field_b200.build as B
    import field_b200.expr as X
    from field_b200.grid import GridMeta
    comp = X.compile_recipe(_recipe(X, length, chain))
    assert (comp.chain is not None) == chain
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    # float32 error of n . x on coordinates below 1.5: four roundings a term, |n|_1 <= sqrt(3) length
    err = 4 * 2.0 ** -24 * 1.5 * np.sqrt(3.0) * max(length, 1.0)
    fb = B.FieldBuilder(comp, meta, guard=max(meta.guard(), err))
    f = fb.build()
    kind, cma = oracle.classify_program(comp.prims, comp.program, meta)
    assert np.array_equal(f.kind.cpu().numpy(), kind)
    assert np.abs(fb.cma.cpu().numpy() - cma).max() <= 1e-5 * meta.pitch + err + 1e-6 * np.abs(cma).max()
    ids = np.where(kind == 0)[0].astype(np.int32)
    want = oracle.tiles_program(comp.prims, comp.program, meta, ids).reshape(len(ids), -1)
    got = f.tiles[:f.n_active].cpu().numpy()
    near = np.abs(want) <= 3 * meta.pitch
    assert np.abs(got - want)[near].max() <= 1e-5 * meta.pitch + err
    assert np.array_equal(got >= 0, want >= 0)
