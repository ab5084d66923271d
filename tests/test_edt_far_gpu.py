"""The x pass's order of strips (the last one first, from six strips a warp on) on smooth masks far from most of the
grid, sites at either end, several nearest sites at the same distance, and axes around the line: equal whole numbers."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [320, 321, 328, 385, 449, 505, 512])
@pytest.mark.parametrize("kind", ["half", "steep", "end", "start", "mirror", "comb"])
def test_far_masks(nx, kind):
    import torch
    import field_b200.edt as E
    shape = (nx, 20, 37)
    x, y, z = np.ogrid[:shape[0], :shape[1], :shape[2]]
    one = np.ones(shape, bool)
    m = {"half": x + y + z < 60, "steep": 7 * x + 3 * y + z > 7 * nx - 300, "end": (x == nx - 1) & (y == 3) & (z % 11 == 0),
         "start": (x == 0) & (z == 36), "mirror": (x == 10) | (x == nx - 11) & (y > 4),
         "comb": (x % 150 == 149) & ((y + z) % 17 == 0)}[kind] & one
    got = E.squared_distance_device(torch.from_numpy(m.view(np.uint8)).cuda(), sites_nonzero=True).cpu().numpy()
    assert np.array_equal(got, oracle.edt_squared(~m))
