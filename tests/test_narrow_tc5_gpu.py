"""The narrow decode products on tcgen05: every cut of K over a cluster, edges of tiles and rows, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def cut(request):
    yield request.param
    from infinilm_b200 import ops
    ops.check_status(torch.device("cuda:0"))


def _rel(got, ref):
    return float((got.double() - ref).abs().amax() / ref.abs().amax())


@pytest.mark.parametrize("cut", [0, 1, 2, 4, 8, -1], indirect=True)
@pytest.mark.parametrize("M,N,K", [(17, 64, 512), (32, 4096, 1024), (33, 70, 576), (40, 200, 640), (48, 33, 1024)])
def test_gated(cuda_device, cut, M, N, K):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()[:, :K]
    w = (torch.randn(2 * N, K, device="cuda", generator=g) * 2 / math.sqrt(K)).bfloat16()
    b = torch.randn(2 * N, device="cuda", generator=g) * 0.1 if M % 2 else None
    sq = (torch.rand(M, 64, device="cuda", generator=g) + 0.5) * 16
    out = torch.full((M, N + 2), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny(x, w, out[:, :N], 0.7, b, glu=1, norm_in=ops.NormedInput(x, sq, 1024, 1e-5), w_static=bool(M % 2), cluster=cut)
    z = 0.7 * torch.rsqrt(sq.double().sum(1, keepdim=True) / 1024 + 1e-5) * (x.double() @ w.double().t()) + (b.double() if b is not None else 0.0)
    ref = z[:, :N] * torch.sigmoid(z[:, :N]) * z[:, N:]
    assert _rel(out[:, :N], ref) <= 2.0 ** -8 and bool(out[:, N:].isnan().all())     # rounded to bfloat16 once


@pytest.mark.parametrize("cut", [0, 1, 2, 4, 8], indirect=True)
@pytest.mark.parametrize("M,N,K", [(17, 512, 64), (31, 1000, 4096), (40, 520, 1024), (48, 1024, 4096), (33, 616, 2560)])
def test_into_the_residual(cuda_device, cut, M, N, K):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).bfloat16()
    b = torch.randn(N, device="cuda", generator=g) if M % 2 else None
    r0, nw = torch.randn(M, N, device="cuda", generator=g), 1 + 0.3 * torch.randn(N, device="cuda", generator=g)
    r, xw, sq = r0.clone(), torch.empty(M, N, device="cuda", dtype=torch.bfloat16), torch.empty(M, (N + 15) // 16, device="cuda")
    ops.gemm_skinny_resid(x, w, 0.6, b, r, 0.35, nw, 1e-5, xw, sq, w_static=True, cluster=cut)
    y = 0.6 * (x.double() @ w.double().t()) + (b.double() if b is not None else 0.0)
    assert float((r.double() - (r0.double() + 0.35 * y)).abs().amax()) <= 2.0 ** -8 * 0.35 * float(y.abs().amax())     # the branch is rounded to bfloat16
    assert _rel(xw, r.double() * nw.double()) <= 2.0 ** -8
    pad = torch.zeros(M, sq.shape[1] * 16, dtype=torch.float64, device="cuda")
    pad[:, :N] = r.double() ** 2
    assert _rel(sq, pad.view(M, -1, 16).sum(-1)) <= 1e-6


@pytest.mark.parametrize("cut", [0, 1, 2, 4, 8], indirect=True)
@pytest.mark.parametrize("nh,nkv,hd", [(16, 2, 64), (4, 1, 128)])
@pytest.mark.parametrize("M,with_cache", [(17, True), (40, True), (48, False)])
def test_rotated_and_stored(cuda_device, cut, nh, nkv, hd, M, with_cache):
    """Against the product in float64, rounded to bfloat16, then rope_store: one bfloat16 step of a rotated value apart, the same slots."""
    from infinilm_b200 import ops
    page, K, N = 16, 576, (nh + 2 * nkv) * hd
    g = torch.Generator().manual_seed(M)
    starts = [(7 * i) % 61 for i in range(M)]
    bt = torch.randperm(M * 4, generator=g).view(M, 4).to(torch.int32).cuda()
    x, w = (torch.randn(M, K, generator=g) * 0.5).bfloat16().cuda(), (torch.randn(N, K, generator=g) * 0.1).bfloat16().cuda()
    bias = torch.randn(N, generator=g).cuda()
    sq = ((torch.rand(M, 33, generator=g) + 0.5) * 10).cuda()
    pos, ent = torch.tensor(starts, dtype=torch.int32).cuda(), torch.arange(M, dtype=torch.int32).cuda()
    inv = (1.0 / (10000.0 ** (torch.arange(hd // 2, dtype=torch.float64) * 2 / hd))).float().cuda()
    z = torch.rsqrt(sq.double().sum(1, keepdim=True) / 528 + 1e-5) * (x.double() @ w.double().t())
    ref = (0.75 * z + bias.double()).bfloat16()
    caches = [torch.zeros(M * 4, 2, nkv, page, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    ops.rope_store(ref, pos, ent, bt, caches[0], page, nh, nkv, hd, hd, inv, 1.1)
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_skinny_rope(x, w, out, 0.75, bias, pos, ent, bt, caches[1] if with_cache else None, page, nh, nkv, hd, hd, inv, 1.1,
                         norm_in=ops.NormedInput(x, sq, 528, 1e-5), w_static=True, cluster=cut)
    scale = float(ref.float().abs().amax())
    assert float((out.float() - ref.float()).abs().amax()) <= 2.0 ** -7 * scale
    if with_cache:
        assert float((caches[0].float() - caches[1].float()).abs().amax()) <= 2.0 ** -7 * scale
        assert torch.equal(caches[0] == 0, caches[1] == 0)
