"""The exported mesh at the block edges around the shared memory a kernel has without asking for more."""
import numpy as np
import pytest

from test_export_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [17, 18, 19, 20, 21, 31])
def test_block_edges_around_the_default_shared_memory(block):
    import field_b200.export as E
    rng = np.random.default_rng(block)
    shp = (2 * block + 1, block, 2 * block - 3)
    noise = rng.normal(size=shp).astype(np.float32)
    _compare(E.marching_cubes_dense(noise, 0.1, pitch=0.5, origin=(1.0, 2.0, 3.0), keys=True, block=block), noise, 0.1,
             (1.0, 2.0, 3.0), 0.5)
