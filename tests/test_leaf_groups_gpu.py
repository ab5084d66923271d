"""Leaf tiles taken in groups of blocks equal those taken one block at a time, bit for bit: short and long
lists, blocks without a stored list, ids that are not active or outside the grid, group sizes up to the
largest and remainders, ring-frame tori, and batches whose groups span recipes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(X, rng, count, size, tori):
    parts = []
    for k in range(count):
        c = rng.uniform(0.05, 0.95, 3) * size
        parts.append((X.sphere(0.04, c), X.box((0.03, 0.05, 0.02), c), X.capsule(c, c + 0.06, 0.015),
                      X.torus(0.3 if tori else 0.05, 0.015, "xyz"[k % 3], c))[k % 4])
    return X.subtract_all(X.union_all(parts), [X.capsule(rng.uniform(0, 1, 3) * size, rng.uniform(0, 1, 3) * size, 0.01)
                                               for _ in range(count // 8)])


@pytest.mark.parametrize("n,block,count,tori", [((160, 150, 141), 4, 60, False), ((120, 120, 120), 4, 1200, False),
                                                ((230, 200, 190), 8, 200, True), ((220, 210, 200), 8, 1500, False)])
def test_groups_equal_single_blocks(n, block, count, tori):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count + block)
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fb = B.FieldBuilder(_recipe(X, rng, count, np.array(n) / max(n), tori), meta)
    fb.classify()
    na = int(fb.count.item())
    assert na >= 6000  # two blocks a group or more
    ids = fb.active[:na].clone()
    for at, bad in ((0, -1), (7, meta.n_blocks), (5003, meta.n_blocks + 5)):  # read as exterior
        ids[at] = bad
    inactive = torch.nonzero(fb.kind != 0).reshape(-1)[:40].to(torch.int32)
    ids[100:100 + len(inactive)] = inactive  # no list of their own
    b3 = block ** 3
    tiles = torch.full((na, b3), 7.0, device="cuda")
    fb.leaf(tiles, na, active=ids)
    one = torch.full((na, b3), 9.0, device="cuda")
    step = 5000  # below what groups start at
    for a in range(0, na, step):
        m = min(step, na - a)
        fb.leaf(one[a:], m, active=ids[a:])
    assert torch.equal(tiles, one)
    for m in (na - 1, na - 3, 12001):  # other remainders; nothing is written past the capacity
        if m <= na:
            part = torch.full((na, b3), 7.0, device="cuda")
            fb.leaf(part, m, active=ids)
            assert torch.equal(part[:m], one[:m]) and bool((part[m:] == 7.0).all())


def test_batch_groups_span_recipes():
    import torch
    import field_b200.batch as BT
    import field_b200.build as B
    import field_b200.expr as X
    rng = np.random.default_rng(4)
    made = []
    for k, n in enumerate((96, 64, 128, 80, 72, 112, 64, 100)):
        count = (700, 5, 40, 300, 1, 90, 900, 12)[k]  # one recipe of a single part; dense ones without lists
        made.append((X.compile_recipe(_recipe(X, rng, count, np.ones(3), k == 3)), BT.cube_meta(n, (4, 4, 8)[k % 3])))
    cap = sum(m.n_blocks * m.block ** 3 for _, m in made)
    bb = BT.BatchBuilder(made, capacity=cap)
    bb.enqueue()
    assert bb.status() == 0
    off, cnt = bb.tile_offsets(), bb.leaf_counts()
    for i, (c, m) in enumerate(made):
        f, single = bb.field(i, off, cnt), B.FieldBuilder(c, m).build()
        assert torch.equal(f.kind, single.kind) and torch.equal(f.tiles, single.tiles[:single.n_active])
    bb.close()
