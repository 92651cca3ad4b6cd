"""Rotation and cache write of many tokens in 16-byte pieces: what the same tokens get a few at a time, and nothing else touched."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rot", [(16, 2, 64, 64), (32, 2, 128, 128), (64, 8, 128, 64), (1, 1, 16, 16), (3, 1, 80, 0), (2, 1, 256, 256), (5, 2, 48, 32)])
@pytest.mark.parametrize("T,cached", [(65, True), (71, False), (131, True)])
def test_many_tokens_as_few_at_a_time(cuda_device, dtype, nh, nkv, hd, rot, T, cached):
    """One to eight tokens a block, the last block with fewer, items beyond a block's threads, a page that is not there."""
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + hd)
    qkv = torch.randn(T, (nh + 2 * nkv) * hd + 8, device="cuda", generator=g).to(dtype)
    pos = (torch.arange(T, device="cuda", dtype=torch.int32) * 7) % 160
    ent = (torch.arange(T, device="cuda", dtype=torch.int32) * 7) // 160
    bt = torch.randperm(80, device="cuda", generator=g).int().view(8, 10)
    bt[0, 3] = -1                                 # nothing is stored for the tokens of this page
    inv = (1.0 / (10000.0 ** (torch.arange(rot // 2, device="cuda", dtype=torch.float64) * 2 / max(rot, 1)))).float() if rot else None
    caches = [torch.full((80, 2, nkv, 16, hd), float("nan"), device="cuda", dtype=dtype) if cached else None for _ in range(2)]
    many, few = qkv.clone(), qkv.clone()
    ops.rope_store(many, pos, ent, bt, caches[0], 16, nh, nkv, hd, rot, inv, 1.1)
    for t in range(0, T, 64):
        ops.rope_store(few[t:t + 64], pos[t:t + 64], ent[t:t + 64], bt, caches[1], 16, nh, nkv, hd, rot, inv, 1.1)
    # x1 c - x2 s with one product rounded, either one: two roundings of at most 1.1 |x|, and the result's own to its type
    bound = 1.1 * 2 * float(qkv.abs().max()) * (2.0 ** -23 if dtype == torch.float32 else 2.0 ** -8)
    assert float((many.float() - few.float()).abs().max()) <= bound and torch.equal(many[:, (nh + nkv) * hd:], qkv[:, (nh + nkv) * hd:])
    if cached:
        assert torch.equal(caches[0].isnan(), caches[1].isnan()) and bool(caches[0].isnan().any())
        assert torch.equal(caches[0][:, 1].nan_to_num(), caches[1][:, 1].nan_to_num())
        for t in range(T):                        # the cache holds the bits of the row
            page = int(bt[ent[t], pos[t] // 16])
            if page >= 0:
                assert torch.equal(caches[0][page, 0, :, pos[t] % 16].reshape(-1), many[t, nh * hd:(nh + nkv) * hd])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rot", [(16, 2, 64, 64), (32, 2, 128, 128), (4, 2, 80, 72)])
def test_rounding_of_a_rotated_pair(cuda_device, dtype, nh, nkv, hd, rot):
    """More than 64 tokens: x1 c - x2 s with x2 s rounded first, x2 c + x1 s with x2 c rounded first, bit for bit in both kernels and types (pairs in
    whole 16-byte pieces or, the last shape in bfloat16, not)."""
    from infinilm_b200 import ops
    T, heads = 200, nh + nkv
    g = torch.Generator(device="cuda").manual_seed(rot)
    pos, ent = (torch.arange(T, device="cuda", dtype=torch.int32) * 37) % 3000, torch.zeros(T, device="cuda", dtype=torch.int32)
    bt = torch.zeros(1, 200, device="cuda", dtype=torch.int32)
    inv = (1.0 / (10000.0 ** (torch.arange(rot // 2, device="cuda", dtype=torch.float64) * 2 / rot))).float()

    def rotated(x):
        ops.rope_store(x, pos, ent, bt, None, 16, nh, nkv, hd, rot, inv, 1.1)
        return x.view(T, nh + 2 * nkv, hd)[:, :heads]
    one = torch.zeros(T, nh + 2 * nkv, hd, device="cuda")
    one[:, :, :rot // 2] = 1
    one = rotated(one.view(T, -1)).double()       # the angles' cosine and sine
    c, s = one[..., :rot // 2], one[..., rot // 2:rot]
    x = torch.randn(T, (nh + 2 * nkv) * hd, device="cuda", generator=g).to(dtype)
    xd = x.view(T, nh + 2 * nkv, hd)[:, :heads].double().clone()
    got = rotated(x)
    x1, x2 = xd[..., :rot // 2], xd[..., rot // 2:rot]
    # products of two float32 are exact in float64; adding rounds them to 53 bits before the rounding to 24, which no pair here is close enough to feel
    assert torch.equal(got[..., :rot // 2], (x1 * c - (x2 * s).float().double()).float().to(dtype))
    assert torch.equal(got[..., rot // 2:rot], ((x2 * c).float().double() + x1 * s).float().to(dtype))
