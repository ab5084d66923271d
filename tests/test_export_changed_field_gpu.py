"""The mesh's second pass over a field that changed since the first: the changes are counted in its error word,
vertex ids stay inside the mesh or are -1, and nothing is written beyond the counted totals -- also where the
first pass left a block's bit words as they were (no crossing)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 4096


def _ball(shape, centre, r):
    import torch
    x, y, z = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float32) for n in shape], indexing="ij")
    return torch.sqrt((x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2) - r


def _tiles(dense, block):
    a, b, c = (n // block for n in dense.shape)
    return dense.reshape(a, block, b, block, c, block).permute(0, 2, 4, 1, 3, 5).reshape(-1, block ** 3).contiguous()


@pytest.mark.parametrize("block", [4, 8, 16, 6])
@pytest.mark.parametrize("change", ["none", "moved", "grown", "noise", "gone"])
def test_second_pass_on_a_changed_field(block, change):
    import torch
    import field_b200._lib as L
    lib = L.lib()
    shape = tuple(n * block for n in (4, 3, 4))
    mid = [n / 2 for n in shape]
    first = _ball(shape, mid, 1.1 * block)
    gen = torch.Generator("cuda").manual_seed(block)
    second = {"none": lambda: first, "moved": lambda: _ball(shape, [mid[0] + 0.6 * block, mid[1], mid[2] - 0.4 * block], 1.1 * block),
              "grown": lambda: first - 0.35 * block, "gone": lambda: first.abs() + 1.0,
              "noise": lambda: torch.randn(shape, device="cuda", generator=gen)}[change]()
    n = 48
    tiles = _tiles(first, block)
    i32 = dict(dtype=torch.int32, device="cuda")
    W, words, st = int(lib.fb_mc_words(block)), int(lib.fb_mc_scan_words(n)), L.stream_handle()
    kind, active, slot = torch.zeros(n, **i32), torch.arange(n, **i32), torch.empty(n, **i32)
    bits = torch.full((n * W,), -1, **i32)  # what a block without a crossing keeps: every bit set
    wpre = torch.full((n * W,), 1 << 28, **i32)
    vcount, tcount = torch.empty(n + 1, **i32), torch.empty(n + 1, **i32)
    totals, scan = torch.empty(2, dtype=torch.int64, device="cuda"), torch.empty(words, **i32)
    args = (kind.data_ptr(), active.data_ptr(), n, tiles.data_ptr(), *shape, block, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0e6)
    assert lib.fb_mc_count_device(*args, slot.data_ptr(), bits.data_ptr(), wpre.data_ptr(), vcount.data_ptr(),
                                  tcount.data_ptr(), totals.data_ptr(), scan.data_ptr(), words, st) == 0
    nv, nt = (int(v) for v in totals.cpu())
    assert nv > 100 and nt > 200
    verts = torch.full((nv + GUARD, 3), 7.0, device="cuda")
    faces = torch.full((nt + GUARD, 3), -7, **i32)
    part, volume, err = (torch.zeros(k, dtype=d, device="cuda") for k, d in
                         ((n, torch.float64), (1, torch.float64), (1, torch.int32)))
    tiles.copy_(_tiles(second, block))
    assert lib.fb_mc_emit_device(*args, slot.data_ptr(), bits.data_ptr(), wpre.data_ptr(), vcount.data_ptr(),
                                 tcount.data_ptr(), verts.data_ptr(), None, faces.data_ptr(), part.data_ptr(),
                                 volume.data_ptr(), err.data_ptr(), st) == 0
    f, e = faces.cpu().numpy(), int(err.item())
    assert (f[nt:] == -7).all() and bool((verts[nv:] == 7.0).all())
    written = f[:nt]
    assert (((written >= -1) & (written < nv)) | (written == -7)).all()
    if change == "none":
        assert e == 0 and (written >= 0).all()
    else:
        assert e > 0
