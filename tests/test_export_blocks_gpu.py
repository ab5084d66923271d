"""The exported mesh on every form of the block kernels (edges 4, 8, 16 and any other), with faces that
need their decision, blocks without a crossing and neighbours without leaves, against the oracle."""
import numpy as np
import pytest

import oracle
from test_export_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [1, 3, 4, 8, 16, 32])
def test_random_and_smooth_fields_on_every_block_edge(block):
    import field_b200.export as E
    rng = np.random.default_rng(block)
    shp = (33, 18, 41)  # ragged for every edge but 1 and 3
    noise = rng.normal(size=shp).astype(np.float32)  # every corner pattern, ambiguous faces among them
    noise[rng.random(shp) < 0.1] = 0.25
    _compare(E.marching_cubes_dense(noise, 0.25, pitch=0.5, origin=(1.0, 2.0, 3.0), keys=True, block=block), noise,
             0.25, (1.0, 2.0, 3.0), 0.5)
    idx = np.indices(shp).reshape(3, -1).T
    ball = (np.linalg.norm(idx - np.array([16, 9, 20]), axis=1) - 7.3).reshape(shp).astype(np.float32)
    nv, nt = _compare(E.marching_cubes_dense(ball, 0.0, pitch=0.25, keys=True, block=block), ball, 0.0, (0.0, 0.0, 0.0),
                      0.25)
    assert nv > 500 and nt > 1000


@pytest.mark.parametrize("block,sign", [(4, 1), (5, -1), (8, 1), (8, -1), (16, 1)])
def test_inactive_neighbours(block, sign):
    """Blocks without leaves among random ones: edges and cubes that enter a block from such a neighbour.
    They all lie on one side, so every crossing has a block with leaves (a field's own guarantee)."""
    import field_b200.export as E
    from field_b200.grid import GridMeta, SparseField
    rng = np.random.default_rng(7 * block)
    meta = GridMeta(0.5, -1.0, 2.0, 0.3, 3 * block + 2, 2 * block, 4 * block - 1, block)
    kind = rng.choice([0, 0, sign], meta.n_blocks).astype(np.int32)
    active = np.where(kind == 0)[0].astype(np.int32)
    tiles = rng.normal(size=(len(active), block, block, block)).astype(np.float32)
    tiles[::3] += 9.0  # leaves without a crossing of their own
    sf = SparseField(meta=meta, kind=kind, active_ids=active, tiles=tiles,
                     corner_min_abs=np.zeros(meta.n_blocks, np.float32))
    dense = oracle.reconstruct(kind, active, tiles, meta)
    nv, nt = _compare(E.marching_cubes(sf, 0.0, keys=True), dense, 0.0, (meta.x0, meta.y0, meta.z0), meta.pitch)
    assert nv > 100 and nt > 100
