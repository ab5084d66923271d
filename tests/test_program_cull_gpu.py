"""General programs pruned per superblock and per block: kinds, corner minima and leaf values are the
float64 oracle's own (rounded once to float32), whatever the tree's operators, kinds, length and grid."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _leaf(X, rng, k):
    c = tuple(rng.uniform(0.1, 0.9, 3))
    if k == 0:
        return X.sphere(float(rng.uniform(0.03, 0.2)), c)
    if k == 1:
        return X.box(tuple(rng.uniform(0.03, 0.2, 3)), c)
    if k == 2:
        return X.capsule(c, tuple(rng.uniform(0.1, 0.9, 3)), float(rng.uniform(0.01, 0.05)))
    if k == 3:
        return X.torus(0.15, 0.04, "xyz"[int(rng.integers(3))], c)
    if k == 4:
        return X.cylinder(0.08, 0.3, axis="xyz"[int(rng.integers(3))], center=c)
    if k == 5:
        return X.cone(0.1, 0.03, 0.25, center=c)
    if k == 6:
        return X.rotate(X.box((0.15, 0.05, 0.08), c), "xyz"[int(rng.integers(3))], float(rng.uniform(10, 80)), about=c)
    if k == 7:
        n = rng.normal(size=3)
        return X.halfspace(tuple(n / np.linalg.norm(n)), float(rng.uniform(-0.2, 0.6)))
    return X.translate(X.scale(X.cross_bore(0.08, 0.0, 0.3), 0.7), *c)


def _tree(X, rng, leaves, ks):
    """A random binary tree: hard and smooth operators of every kind, offsets in between."""
    if leaves == 1:
        return _leaf(X, rng, int(rng.integers(0, 9)))
    left = int(rng.integers(1, leaves))
    a, b = _tree(X, rng, left, ks), _tree(X, rng, leaves - left, ks)
    op = (X.union, X.union, X.subtract, X.intersect)[int(rng.integers(4))]
    t = op(a, b, k=float(rng.choice(ks)))
    return X.offset(t, float(rng.uniform(-0.02, 0.02))) if rng.random() < 0.2 else t


# leaves past 128 make programs longer than a pruned one may be (256 instructions) before pruning
@pytest.mark.parametrize("leaves,ks,n,block,seed", [
    (3, (0.0,), (9, 8, 7), 4, 0), (12, (0.0,), (65, 64, 33), 8, 1), (12, (0.0, 0.03), (70, 41, 64), 4, 2),
    (40, (0.0, 0.05), (50, 66, 49), 16, 3), (200, (0.0,), (64, 48, 33), 8, 4), (180, (0.0, 0.02), (40, 40, 40), 4, 5),
    (25, (0.02, 0.1), (130, 36, 36), 8, 6)])
def test_pruned_programs_equal_the_oracle(leaves, ks, n, block, seed):
    import field_b200.build as B
    import field_b200.expr as X
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(seed)
    # a root that is no chain: an intersection with a union of subtrees
    t = X.intersect(X.sphere(0.48, (0.5, 0.5, 0.5)), X.union(_tree(X, rng, leaves, ks), X.subtract(
        _tree(X, rng, 2, ks), _tree(X, rng, 2, ks))))
    comp = X.compile_recipe(t)
    assert comp.chain is None
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fb = B.FieldBuilder(comp, meta)
    f = fb.build()
    kind, cma = oracle.classify_program(comp.prims, comp.program, meta)
    assert np.array_equal(f.kind.cpu().numpy(), kind)
    assert np.array_equal(fb.cma.cpu().numpy(), cma.astype(np.float32))
    active = np.where(kind == 0)[0].astype(np.int32)
    assert f.n_active == len(active) > 0
    want = oracle.tiles_program(comp.prims, comp.program, meta, active).reshape(len(active), -1).astype(np.float32)
    assert np.array_equal(f.tiles[:f.n_active].cpu().numpy(), want)
    # blocks without a program of their own (shifted ids) walk the whole one
    shifted = np.minimum(active + 1, meta.n_blocks - 1).astype(np.int32)
    import torch
    tiles = torch.empty_like(f.tiles)
    act = fb.active.clone()
    act[:len(active)] = torch.from_numpy(shifted).cuda()
    fb.leaf(tiles, f.n_active, active=act)
    want = oracle.tiles_program(comp.prims, comp.program, meta, shifted).reshape(len(active), -1).astype(np.float32)
    assert np.array_equal(tiles[:f.n_active].cpu().numpy(), want)
