"""Accelerated queries over steps from far below a voxel to beyond the grid, points inside and far outside it, and
chains from one element up: every path's values and gradients are the whole chain's, bit for bit, also with
scratch sized without the step and with none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(X, rng, count, kind):
    t = X.sphere(0.3, (0.5, 0.4, 0.3))
    for i in range(count - 1):
        c = rng.uniform(0.05, 0.9, 3)
        p = (X.sphere(0.06, c), X.box((0.03, 0.06, 0.05), c), X.capsule(c, c + 0.1, 0.02), X.torus(0.06, 0.02, "y", c))[i % 4]
        if kind == "run":
            t = X.union(t, p)
        elif kind == "alternate":
            t = X.subtract(t, p) if i % 2 else X.union(t, p)
        else:
            t = X.union(t, p, k=0.03)
    return t


@pytest.mark.parametrize("count,kind", [(1, "run"), (3, "run"), (1100, "run"), (1100, "alternate"), (12, "run"), (13, "alternate"), (90, "run"),
                                        (300, "run"), (90, "alternate"), (90, "blend"), (300, "blend")])
@pytest.mark.parametrize("n,block", [((64, 40, 50), 8), ((200, 96, 130), 8), ((33, 20, 9), 4)])
def test_steps_and_points(count, kind, n, block):
    import torch
    import field_b200._lib as L
    import field_b200.build as B
    import field_b200.expr as X
    import field_b200.query as Q
    from field_b200.grid import GridMeta
    rng = np.random.default_rng(count)
    comp = X.compile_recipe(_recipe(X, rng, count, kind))
    assert comp.chain is not None
    pitch = 1.0 / max(n)
    meta = GridMeta(0.0, 0.0, 0.0, pitch, *n, block)
    fb = B.FieldBuilder(comp, meta)
    fb.classify()
    plain, fast = Q.RecipeQueries(comp), Q.RecipeQueries(comp, builder=fb)
    size = np.array(n) * pitch
    pts = rng.uniform(-0.1, 1.1, (45000, 3)) * size
    pts[5::7] = rng.uniform(-2.0, 3.0, (len(pts[5::7]), 3)) * size  # far outside, scattered
    pts[3] = np.nan
    pts[4] = 1e30
    pts = torch.from_numpy(pts.astype(np.float32)).cuda()
    same = lambda a, b: torch.equal(a.nan_to_num(nan=1e30), b.nan_to_num(nan=1e30))
    edge = (32 if max(n) > 128 else 16) * pitch  # a superblock's
    lib = L.lib()
    for m in (1, 300, 3000, 45000):
        p = pts[:m].contiguous()
        assert same(plain.values(p), fast.values(p)), m
        for h in (pitch, 0.2499 * edge, 0.2501 * edge, -0.7 * edge, 0.4, 5.0):
            v0, g0 = plain.values_and_gradients(p, h=h)
            v1, g1 = fast.values_and_gradients(p, h=h)
            assert same(v0, v1) and same(g0, g1), (m, h)
            g2 = torch.empty_like(g0)
            fast._run(p, None, g2, h=h)
            assert same(g0, g2), (m, h)
    # the C entry with the step-less scratch, and with none
    a, h = fast._accel, 0.4
    for m in (3000, 45000):
        p = pts[:m].contiguous()
        v0, g0 = plain.values_and_gradients(p, h=h)
        for nbytes in (int(lib.fb_query_scratch_bytes(a[4].ctypes.data, m, 1)), 0):
            scratch = torch.empty(max(nbytes, 1), dtype=torch.uint8, device="cuda")
            v1, g1 = torch.empty_like(v0), torch.empty_like(g0)
            assert lib.fb_query_points_device(
                fast.primf.data_ptr(), fast.chain.data_ptr(), fast.n_chain, 1, a[0], a[1], a[2], a[3].ctypes.data,
                a[4].ctypes.data, *a[5], p.data_ptr(), m, h, v1.data_ptr(), g1.data_ptr(),
                scratch.data_ptr() if nbytes else None, nbytes, L.stream_handle()) == 0
            assert same(v0, v1) and same(g0, g1), (m, nbytes)
