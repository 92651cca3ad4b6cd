"""How many splits of the keys a decode step takes: one for a few pages of small heads, else what fills the device (no GPU)."""
import pytest
import torch

from infinilm_b200.parts.attention import PagedAttend


@pytest.mark.parametrize("nh,nkv,hd", [(32, 2, 128), (32, 8, 128), (16, 4, 96), (8, 2, 256), (12, 12, 80)])
@pytest.mark.parametrize("pages,requests", [(5, 1), (8, 4), (16, 1), (16, 8)])
def test_heads_beyond_64_keep_their_splits(nh, nkv, hd, pages, requests):
    core = PagedAttend(torch.bfloat16, nh, nkv, hd, hd ** -0.5)
    base, resident = requests * nkv, 444
    assert core.decode_splits(base, pages, resident) == max(1, min(296 // base, (pages + 3) // 4))


@pytest.mark.parametrize("hd", [16, 32, 48, 64])
def test_a_few_pages_of_small_heads_are_one_split(hd):
    core = PagedAttend(torch.bfloat16, 16, 2, hd, hd ** -0.5)
    assert [core.decode_splits(2, p, 444) for p in (1, 5, 16, 17)] == [1, 1, 1, 5]
