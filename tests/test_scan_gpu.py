"""The shared exclusive scan at the edges of its tiles and of the direct form (4096 tiles), through the tree's
per-word rank tables."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [2, 4095, 4096, 4097, 3 * 4096, 5 * 4096 + 17, 4096 * 4096, 4096 * 4096 + 1])
def test_rank_tables_are_exclusive_prefix_sums(entries):
    import torch
    import field_b200._lib as L
    lib = L.lib()
    words = entries - 1  # the tables hold one entry more
    nodes = 16 * words
    gen = torch.Generator("cuda").manual_seed(entries)
    packed = torch.randint(-2 ** 31, 2 ** 31 - 1, (words,), dtype=torch.int32, device="cuda", generator=gen)
    two, three = (torch.full((entries,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    scratch = torch.empty(int(lib.fb_tree_rank_words_scratch_bytes(nodes)), dtype=torch.uint8, device="cuda")
    assert lib.fb_tree_rank_words_device(packed.data_ptr(), nodes, two.data_ptr(), three.data_ptr(), scratch.data_ptr(),
                                         scratch.numel(), L.stream_handle()) == 0
    n2, n3 = torch.zeros(words, dtype=torch.int32, device="cuda"), torch.zeros(words, dtype=torch.int32, device="cuda")
    for k in range(16):
        code = (packed >> (2 * k)) & 3
        n2 += code == 2
        n3 += code == 3
    zero = torch.zeros(1, dtype=torch.int64, device="cuda")
    for got, counts in ((two, n2), (three, n3)):
        assert torch.equal(got.long(), torch.cat([zero, torch.cumsum(counts, 0)]))
