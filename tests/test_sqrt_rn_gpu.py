"""The canonical float32 forms' square root equals the IEEE root on every non-negative float."""
import pytest

pytestmark = pytest.mark.gpu


def test_sqrt_rn_equals_the_ieee_root_everywhere():
    import torch
    import field_b200._lib as L
    lib = L.lib()
    step = 1 << 26
    out = torch.empty(step, dtype=torch.float32, device="cuda")
    for lo in range(0, 0x7f800000, step):  # +0 up to the largest finite float, subnormals among them
        bits = torch.arange(lo, min(lo + step, 0x7f800001), dtype=torch.int32, device="cuda")  # ... and infinity
        x = bits.view(torch.float32)
        assert lib.fb_sqrt_rn_probe(x.data_ptr(), out.data_ptr(), x.numel(), L.stream_handle()) == 0
        assert torch.equal(out[:x.numel()].view(torch.int32), torch.sqrt(x).view(torch.int32)), hex(lo)
    x = torch.tensor([float("nan")], device="cuda")
    assert lib.fb_sqrt_rn_probe(x.data_ptr(), out.data_ptr(), 1, L.stream_handle()) == 0
    assert bool(torch.isnan(out[0]))
