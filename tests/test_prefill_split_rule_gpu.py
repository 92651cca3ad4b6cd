"""Which blocks of the prompt attention share their keys with a second one follows from their own keys: the same bits beside a longer request, with a
wider block table, and in an eager step and a replayed one."""
import math

import pytest
import torch

from replay_util import build_engine
from tiny_configs import make_weights, random_ids, tiny_d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,hd,start,q", [(8, 1, 64, 0, 300), (8, 2, 64, 430, 90), (8, 2, 64, 600, 40), (4, 1, 128, 900, 150), (4, 1, 128, 950, 100), (4, 1, 128, 1900, 90)])
def test_bits_do_not_follow_the_table(cuda_device, nh, nkv, hd, start, q):
    """Chains below, across and above the tile from which keys are shared; tables as wide as the request, of 2,048 keys, and beside one of 6,000."""
    from infinilm_b200 import ops
    n, pages = start + q, (start + q + 15) // 16
    g = torch.Generator(device="cuda").manual_seed(n)
    cache = torch.randn(380, 2, nkv, 16, hd, device="cuda", generator=g).bfloat16()
    rows = (torch.randn(q, (nh + 2 * nkv) * hd, device="cuda", generator=g) * 2).bfloat16()
    order = torch.randperm(380, generator=torch.Generator().manual_seed(1)).int()
    kv_map, tpt, outs = ops.kv_tensor_map(cache), ops.prefill_tc5_rows(hd) // (nh // nkv), []
    for width, lens in ((pages, [n]), (max(pages, 128), [n]), (375, [n, 6000])):
        bt = torch.full((len(lens), width), -1, dtype=torch.int32)
        bt[0, :pages] = order[:pages]
        if len(lens) > 1:
            bt[1, :375] = order[:375]
        T = q + 3 * (len(lens) - 1)               # (the long request brings three tokens)
        qkv = rows if len(lens) == 1 else torch.cat([rows, rows[:3]])
        out = torch.full((T, nh * hd), float("nan"), device="cuda", dtype=torch.bfloat16)
        tiles = -(-q // tpt) + len(lens) - 1
        ops.attention_prefill_tc5(qkv, out, kv_map, bt.cuda(), torch.tensor([0, q, T][:len(lens) + 1], dtype=torch.int32).cuda(),
                                  torch.tensor(lens, dtype=torch.int32).cuda(), 0, len(lens), tiles, 16, nh, nkv, hd, 1 / math.sqrt(hd), None)
        outs.append(out[:q])
    ops.check_status("cuda:0")
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("extra", [0, 5])
def test_a_bound_on_the_tiles_decides_as_given(cuda_device, extra):
    """296 blocks are shared, 301 by the bound are not, however many are launched for the same tokens."""
    from infinilm_b200 import ops
    nh, nkv, hd, q = 8, 1, 64, 296 * 16
    g = torch.Generator(device="cuda").manual_seed(extra)
    cache = torch.randn(300, 2, nkv, 16, hd, device="cuda", generator=g).bfloat16()
    qkv = (torch.randn(q, (nh + 2 * nkv) * hd, device="cuda", generator=g) * 2).bfloat16()
    bt, outs = torch.arange(296, dtype=torch.int32).view(1, -1).cuda(), []
    for tiles in (296, 301):
        out = torch.full((q, nh * hd), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.attention_prefill_tc5(qkv, out, ops.kv_tensor_map(cache), bt, torch.tensor([0, q], dtype=torch.int32).cuda(), torch.tensor([q], dtype=torch.int32).cuda(),
                                  0, 1, tiles, 16, nh, nkv, hd, 1 / math.sqrt(hd), None, n_tiles_rule=296 + extra)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("hd,n", [(64, 490), (64, 511), (64, 700), (128, 1010), (128, 2000), (128, 2050)])
def test_eager_and_replayed_steps_agree_in_bfloat16(cuda_device, hd, n):
    """A whole prompt as one portion: eager twice, then with its key's bounds, captured and replayed."""
    from infinilm_b200.engine import StepEntry
    raw = dict(tiny_d(), head_dim=hd, max_position_embeddings=4096)
    raw["rope_scaling"] = dict(raw["rope_scaling"], short_factor=[1.0 + 0.01 * i for i in range(hd // 2)],
                               long_factor=[2.0 + 0.01 * i for i in range(hd // 2)], original_max_position_embeddings=4096)
    eng = build_engine(raw, make_weights(raw, 3), "bfloat16", num_pages=140, max_batch_tokens=2200)
    eng.enable_graphs()
    ids, outs = random_ids(n, raw["vocab_size"], n), []
    for k in range(6):
        seq = eng.open(k)
        outs.append(eng.step([StepEntry(seq, ids, [n - 1])]).clone())
        eng.close(seq)
    assert eng.runner.portion_replays > 0
    assert all(torch.equal(outs[0], o) for o in outs[1:])
