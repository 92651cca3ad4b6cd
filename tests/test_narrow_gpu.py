"""The fused decode products of 17 to 48 rows on a narrow model against float64, and against the kernels they stand for."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, ref):
    return float((got.double() - ref).abs().amax() / ref.abs().amax())


@pytest.mark.parametrize("M", [17, 24, 25, 32, 33, 40, 41, 48])
@pytest.mark.parametrize("N,K", [(8, 512), (70, 520), (4096, 1024), (33, 1016)])
@pytest.mark.parametrize("act", [1, 2, 3])
def test_gated(cuda_device, M, N, K, act):
    from infinilm_b200 import ops
    if act > 1 and N == 4096:
        pytest.skip("one gate at the largest size")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * N, K, device="cuda", generator=g) * 2 / math.sqrt(K)).bfloat16()
    b = torch.randn(2 * N, device="cuda", generator=g) * 0.1 if M % 2 else None
    sq = (torch.rand(M, 64, device="cuda", generator=g) + 0.5) * 16
    ni = ops.NormedInput(x, sq, 1024, 1e-5)
    outs = []
    for static in (False, True):
        out = torch.full((M, N + 2), float("nan"), device="cuda", dtype=torch.bfloat16)
        ops.gemm_skinny(x, w, out[:, :N], 0.7, b, glu=act, norm_in=ni, act_params=(7.0, 1.7), w_static=static)
        outs.append(out)
    z = 0.7 * torch.rsqrt(sq.double().sum(1, keepdim=True) / 1024 + 1e-5) * (x.double() @ w.double().t()) + (b.double() if b is not None else 0.0)
    p, u = z[:, :N], z[:, N:]
    if act == 1:
        ref = p * torch.sigmoid(p) * u
    elif act == 2:
        ref = torch.nn.functional.gelu(p, approximate="tanh") * u
    else:
        p = p.clamp(max=7.0)
        ref = p * torch.sigmoid(1.7 * p) * (u.clamp(-7.0, 7.0) + 1)
    assert _rel(outs[0][:, :N], ref) <= 2.0 ** -8          # rounded to bfloat16 once: half a step, and as much for f32 sums and the fast units
    assert torch.equal(outs[0][:, :N], outs[1][:, :N]) and bool(outs[0][:, N:].isnan().all())


@pytest.mark.parametrize("M", [17, 24, 25, 32, 33, 48])
@pytest.mark.parametrize("N,K", [(512, 8), (520, 1024), (1000, 1032), (1024, 4096), (616, 2560)])
def test_into_the_residual(cuda_device, M, N, K):
    from infinilm_b200 import ops
    if not ops.skinny_resid_ok(M, K, N):
        assert M > ops.NARROW_LONG_ROWS and K > ops.NARROW_WIDTH
        pytest.skip("the library's")
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).bfloat16()
    b = torch.randn(N, device="cuda", generator=g) if M % 2 else None
    resid0, nw = torch.randn(M, N, device="cuda", generator=g), 1 + 0.3 * torch.randn(N, device="cuda", generator=g)
    y = 0.6 * (x.double() @ w.double().t()) + (b.double() if b is not None else 0.0)
    outs = []
    for static in (False, True):
        r, xw, sq = resid0.clone(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, (N + 15) // 16, device="cuda")
        ops.gemm_skinny_resid(x, w, 0.6, b, r, 0.35, nw, 1e-5, xw, sq, w_static=static)
        outs.append((r, xw, sq))
    r, xw, sq = outs[0]
    assert all(torch.equal(a, c) for a, c in zip(*outs))
    assert float((r.double() - (resid0.double() + 0.35 * y)).abs().amax()) <= 2.0 ** -8 * 0.35 * float(y.abs().amax())     # the branch is rounded to bfloat16
    assert _rel(xw, r.double() * nw.double()) <= 2.0 ** -8
    pad = torch.zeros(M, sq.shape[1] * 16, dtype=torch.float64, device="cuda")
    pad[:, :N] = r.double() ** 2
    assert _rel(sq, pad.view(M, -1, 16).sum(-1)) <= 1e-6


@pytest.mark.parametrize("nh,nkv,hd,rot", [(16, 2, 64, 64), (3, 1, 48, 16), (2, 2, 32, 0)])
@pytest.mark.parametrize("M", [17, 40, 48])
def test_rotated_and_stored(cuda_device, nh, nkv, hd, rot, M):
    """Against the product alone in float64, rounded to bfloat16, then rope_store: one bfloat16 step of a rotated value apart, the same slots."""
    from infinilm_b200 import ops
    page, K = 16, 520
    N = (nh + 2 * nkv) * hd
    g = torch.Generator().manual_seed(M)
    starts = [(7 * i) % 61 for i in range(M)]
    bt = torch.randperm(M * 4, generator=g).view(M, 4).to(torch.int32).cuda()
    x = (torch.randn(M, K, generator=g) * 0.5).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) * 0.1).bfloat16().cuda()
    bias = torch.randn(N, generator=g).cuda()
    pos, ent = torch.tensor(starts, dtype=torch.int32).cuda(), torch.arange(M, dtype=torch.int32).cuda()
    inv = (1.0 / (10000.0 ** (torch.arange(rot // 2, dtype=torch.float64) * 2 / max(rot, 1)))).float().cuda() if rot else None
    ref = (0.75 * (x.double() @ w.double().t()) + bias.double()).bfloat16()
    caches = [torch.zeros(M * 4, 2, nkv, page, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    ops.rope_store(ref, pos, ent, bt, caches[0], page, nh, nkv, hd, rot, inv, 1.1)
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny_rope(x, w, out, 0.75, bias, pos, ent, bt, caches[1], page, nh, nkv, hd, rot, inv, 1.1, w_static=True)
    scale = float(ref.float().abs().amax())
    assert float((out.float() - ref.float()).abs().amax()) <= 2.0 ** -7 * scale
    assert float((caches[0].float() - caches[1].float()).abs().amax()) <= 2.0 ** -7 * scale
    assert torch.equal(caches[0] == 0, caches[1] == 0)


@pytest.mark.parametrize("K", [512, 1016, 1024])
@pytest.mark.parametrize("M", [17, 24, 32, 33, 48])
@pytest.mark.parametrize("with_cache,with_bias", [(True, True), (False, True), (True, False)])
def test_rotated_rows_whose_norm_is_unfinished(cuda_device, M, K, with_cache, with_bias):
    """Rows whose 1/rms differ by orders of magnitude, up to the widest model: row by row against float64, rounded to bfloat16 and then rotated."""
    from infinilm_b200 import ops
    nh, nkv, hd, rot, page = 4, 2, 64, 32, 16
    N = (nh + 2 * nkv) * hd
    g = torch.Generator().manual_seed(M + K)
    pos = torch.tensor([(11 * i) % 63 for i in range(M)], dtype=torch.int32)
    bt = torch.randperm(M * 4, generator=g).view(M, 4).to(torch.int32).cuda()
    x = torch.randn(M, K, generator=g).bfloat16()
    w = (torch.randn(N, K, generator=g) / math.sqrt(K)).bfloat16()
    bias = torch.randn(N, generator=g) * 1e-3 if with_bias else None
    sq = (torch.rand(M, 64, generator=g) + 0.5) * 10.0 ** (torch.arange(M).view(M, 1) % 7 - 3).float()
    inv = (1.0 / (10000.0 ** (torch.arange(rot // 2, dtype=torch.float64) * 2 / rot))).float()
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    cache = torch.zeros(M * 4, 2, nkv, page, hd, dtype=torch.bfloat16, device="cuda") if with_cache else None
    ops.gemm_skinny_rope(x.cuda(), w.cuda(), out, 0.75, None if bias is None else bias.cuda(), pos.cuda(), torch.arange(M, dtype=torch.int32).cuda(), bt, cache, page,
                         nh, nkv, hd, rot, inv.cuda(), 1.1, norm_in=ops.NormedInput(x.cuda(), sq.cuda(), 1024, 1e-5))
    y = 0.75 * torch.rsqrt(sq.double().sum(1, keepdim=True) / 1024 + 1e-5) * (x.double() @ w.double().t()) + (bias.double() if bias is not None else 0.0)
    y = y.view(M, nh + 2 * nkv, hd)
    ang = pos.double().view(M, 1, 1) * inv.double()
    lo, hi = y[..., :rot // 2], y[..., rot // 2:rot]
    turned = torch.cat([(lo * ang.cos() - hi * ang.sin()) * 1.1, (hi * ang.cos() + lo * ang.sin()) * 1.1, y[..., rot:]], -1)
    ref = torch.cat([turned[:, :nh + nkv], y[:, nh + nkv:]], 1)
    got = out.cpu().double().view(M, nh + 2 * nkv, hd)
    # two roundings to bfloat16 of values within the head's largest (the second of two rotated ones), and the angle's rounding (63 radians: 63 x 2^-23 at most)
    assert bool(((got - ref).abs() <= 3 * 2.0 ** -8 * ref.abs().amax(-1, keepdim=True)).all())
    if with_cache:
        for m in range(M):
            p = int(bt[m, int(pos[m]) // page])
            assert torch.equal(cache[p, 0, :, int(pos[m]) % page].cpu(), out[m].view(-1, hd)[nh:nh + nkv].cpu())
            assert torch.equal(cache[p, 1, :, int(pos[m]) % page].cpu(), out[m].view(-1, hd)[nh + nkv:].cpu())
        assert int((cache != 0).any(-1).sum()) == 2 * nkv * M


def test_step_with_and_without_the_norm_in_its_products(cuda_device):
    """A model 512 wide in portions of 17 to 48 rows, with rows either side of them, against the plain model, with the fused products and with the kernels
    they stand for."""
    from infinilm_b200 import ops
    from infinilm_b200.parts.blocks import PreNormResidual
    from replay_util import TOL, build_engine, first_bad_row, plain_logits, rel_err, run_cut
    from tiny_configs import TINY, make_weights, random_ids
    raw = dict(TINY["d"](), hidden_size=512, intermediate_size=1288)
    w = make_weights(raw, 6)
    cuts = [17, 16, 33, 48, 49, 32, 1, 25]
    ids = random_ids(sum(cuts), raw["vocab_size"], 78)
    ref = plain_logits(raw, w, ids, "bfloat16")
    was = PreNormResidual.FUSE_NORM
    try:
        for fuse in (False, True):
            PreNormResidual.FUSE_NORM = fuse
            eng = build_engine(raw, w, "bfloat16")
            got = run_cut(eng, ids, cuts)
            bad = first_bad_row(got, ref, TOL["bfloat16"])
            assert bad is None, f"fuse={fuse}: first wrong position {bad} (rel err {rel_err(got[bad], ref[bad]):.2e})"
    finally:
        PreNormResidual.FUSE_NORM = was
    for b in eng.model.blocks:
        for T in cuts:
            assert (b.mixer.fuses_tail(T) and b.mixer.accepts_normed(T) and b.ffn.accepts_normed(T)) == (T <= ops.NARROW_MAX_ROWS)
            assert b.ffn.fuses_tail(T) == (T <= ops.NARROW_LONG_ROWS)      # 1,288 columns into the residual
