"""Prompt attention whose key tiles two blocks of a cluster share, against the plain kernel: from eight (heads of 128: 17) tiles of 64 on, and up to one block a place on the device."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,hd", [(8, 1, 64), (3, 3, 64), (7, 1, 128)])
@pytest.mark.parametrize("starts,qlens", [([0, 0, 0, 2040], [192, 193, 256, 9]), ([190, 255, 1000, 2045], [3, 66, 9, 3])])
@pytest.mark.parametrize("window,sunk", [(None, False), (None, True), (150, False), (300, True)])
def test_halves_of_the_keys(cuda_device, nh, nkv, hd, starts, qlens, window, sunk):
    _compare(nh, nkv, hd, starts, qlens, window, sunk)


@pytest.mark.parametrize("over", [0, 1])
def test_as_many_blocks_as_the_device_holds_and_one_more(cuda_device, over):
    """Heads of 64, sixteen tokens a block: 296 blocks are split, 297 are not."""
    _compare(8, 1, 64, [500, 0], [16 * 295 + over, 16], 700, False)


def _compare(nh, nkv, hd, starts, qlens, window, sunk):
    from infinilm_b200 import ops
    lens = [s + q for s, q in zip(starts, qlens)]
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    n_pages = [(n + 15) // 16 for n in lens]
    bt, perm, k = torch.full((len(lens), max(n_pages)), -1, dtype=torch.int32), torch.randperm(sum(n_pages)), 0
    for e, n in enumerate(n_pages):
        bt[e, :n] = perm[k:k + n]
        k += n
    bt, T = bt.cuda(), sum(qlens)
    cache = torch.randn(k, 2, nkv, 16, hd, device="cuda", generator=g).bfloat16()
    qkv = (torch.randn(T, (nh + 2 * nkv) * hd, device="cuda", generator=g) * 2).bfloat16()
    sink = torch.randn(nh, device="cuda", generator=g) if sunk else None
    pos = torch.cat([torch.arange(s, s + q) for s, q in zip(starts, qlens)]).int().cuda()
    ent = torch.cat([torch.full((q,), e) for e, q in enumerate(qlens)]).int().cuda()
    qstart = torch.tensor([0] + torch.tensor(qlens).cumsum(0).tolist(), dtype=torch.int32).cuda()
    ref, out = torch.empty(T, nh * hd, device="cuda", dtype=torch.bfloat16), torch.full((T, nh * hd), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.attention_plain(qkv, ref, cache, bt, pos, ent, 16, nh, nkv, hd, 1 / math.sqrt(hd), window, sink=sink)
    tpt = ops.prefill_tc5_rows(hd) // (nh // nkv)
    ops.attention_prefill_tc5(qkv, out, ops.kv_tensor_map(cache), bt, qstart, torch.tensor(lens, dtype=torch.int32).cuda(), 0, len(lens),
                              sum(-(-q // tpt) for q in qlens), 16, nh, nkv, hd, 1 / math.sqrt(hd), window, sink=sink)
    torch.cuda.synchronize()
    ops.check_status("cuda:0")
    # probabilities and two results rounded to bfloat16, each within 2^-9 of values up to the largest of v
    assert float((out.float() - ref.float()).abs().max()) <= 3 * 2.0 ** -9 * float(cache[:, 1].float().abs().max())
