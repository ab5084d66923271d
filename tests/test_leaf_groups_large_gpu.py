"""Leaf tiles where blocks go in groups (many blocks of short lists) and where they do not (long lists, fewer blocks)
equal those taken one block at a time, bit for bit: around the least count, with ids that are not active or outside
the grid, and over a batch's recipes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(X, rng, count, size, scale, tori=False):
    parts = []
    for k in range(count):
        c = rng.uniform(0.05, 0.95, 3) * size
        parts.append((X.sphere(0.3 * scale, c), X.box(np.array((0.2, 0.3, 0.15)) * scale, c), X.capsule(c, c + 0.4 * scale, 0.1 * scale),
                      X.torus(0.4 if tori else 0.3 * scale, 0.06 * scale, "xyz"[k % 3], c))[k % 4])
    return X.subtract_all(X.union_all(parts), [X.capsule(rng.uniform(0, 1, 3) * size, rng.uniform(0, 1, 3) * size, 0.02)
                                               for _ in range(max(count // 8, 1))])


@pytest.mark.parametrize("n,block,count,scale,tori,short", [
    ((300, 290, 281), 4, 30, 0.8, False, True), ((390, 400, 380), 8, 40, 1.0, True, True),
    ((250, 250, 240), 4, 4000, 0.25, False, False), ((300, 290, 281), 4, 300, 0.3, False, None)])
def test_groups_equal_single_blocks(n, block, count, scale, tori, short):
    import torch
    import field_b200.build as B
    import field_b200.expr as X
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count + block)
    meta = GridMeta(0.0, 0.0, 0.0, 1.0 / max(n), *n, block)
    fb = B.FieldBuilder(_recipe(X, rng, count, np.array(n) / max(n), scale, tori), meta)
    fb.classify()
    na = int(fb.count.item())
    if short is not None:
        assert na >= 40000
    ids = fb.active[:na].clone()
    for at, bad in ((0, -1), (7, meta.n_blocks), (20003, meta.n_blocks + 5)):  # read as exterior
        ids[at] = bad
    inactive = torch.nonzero(fb.kind != 0).reshape(-1)[:40].to(torch.int32)
    ids[100:100 + len(inactive)] = inactive  # no list of their own
    b3 = block ** 3
    one = torch.full((na, b3), 9.0, device="cuda")
    for a in range(0, na, 20000):  # below what groups start at
        fb.leaf(one[a:], min(20000, na - a), active=ids[a:])
    for m in {na, na - 1, na - 3, 40001, 40000, 39999}:  # nothing is written past the capacity
        if m <= na:
            part = torch.full((na, b3), 7.0, device="cuda")
            fb.leaf(part, m, active=ids)
            assert torch.equal(part[:m], one[:m]) and bool((part[m:] == 7.0).all()), m


@pytest.mark.parametrize("counts", [(20, 1, 40, 12), (1500, 900, 2000, 3)])
def test_batch(counts):
    import torch
    import field_b200.batch as BT
    import field_b200.build as B
    import field_b200.expr as X
    rng = np.random.default_rng(5)
    made = []
    for k, (n, block) in enumerate(((200, 4), (330, 8), (180, 4), (300, 8))):
        scale = 0.8 if counts[k] < 100 else 0.2
        made.append((X.compile_recipe(_recipe(X, rng, counts[k], np.ones(3), scale)), BT.cube_meta(n, block)))
    bb = BT.BatchBuilder(made, capacity=sum(m.n_blocks * m.block ** 3 for _, m in made))
    for _ in range(2):
        bb.enqueue()
        assert bb.status() == 0
        off, cnt = bb.tile_offsets(), bb.leaf_counts()
        for i, (c, m) in enumerate(made):
            f, single = bb.field(i, off, cnt), B.FieldBuilder(c, m).build()
            assert torch.equal(f.kind, single.kind) and torch.equal(f.tiles, single.tiles[:single.n_active])
    bb.close()
