"""Products over many groups of a few rows: every tile finds its group, among up to hundreds, and a row has the same bits in any tile."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layout(G, M, seed):
    """Groups of 0 to 2 rows, one of 16, one of 17 and the last of the rest."""
    g = torch.Generator().manual_seed(seed)
    counts = torch.randint(0, 3, (G,), generator=g)
    counts[G // 2], counts[G // 3] = 16, 17
    counts[-1] = 0
    over = int(counts.sum()) - M
    for i in range(G):
        cut = min(max(over, 0), int(counts[i])) if i not in (G // 2, G // 3) else 0
        counts[i] -= cut
        over -= cut
    counts[-1] += max(-over, 0)
    return torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)])


@pytest.mark.parametrize("G,M", [(12, 48), (63, 100), (64, 100), (65, 70), (128, 300), (300, 330)])
@pytest.mark.parametrize("N,K,glu", [(40, 96, True), (72, 1408, False), (130, 64, True)])
def test_ragged(cuda_device, G, M, N, K, glu):
    from infinilm_b200 import ops
    off = _layout(G, M, G + N)
    M = int(off[-1])
    assert M <= 4 * G                                      # few rows a group
    g = torch.Generator().manual_seed(K)
    a = torch.randn(M + 3, K, generator=g).bfloat16()
    w = (torch.randn(G, (2 if glu else 1) * N, K, generator=g) * 2 / math.sqrt(K)).bfloat16()
    rows = torch.randint(0, M + 3, (M,), generator=g, dtype=torch.int32)
    scale = 0.5 + torch.rand(M + 3, generator=g)
    out = torch.full((M + 1, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(a.cuda(), w.cuda(), out[:M], group_off=off.to(torch.int32).cuda(), a_rows=rows.cuda(), n_rows=M, glu=glu, row_scale=scale.cuda())
    for e in range(G):
        lo, hi = int(off[e]), int(off[e + 1])
        if lo == hi:
            continue
        r = rows[lo:hi].long()
        y = (a[r].double() @ w[e].double().t()) * scale[r].double()[:, None]
        if glu:
            gt, up = y[:, :N].bfloat16().double(), y[:, N:].bfloat16().double()
            y = gt * torch.sigmoid(gt) * up
        # rounded to bfloat16 once; with a gate its two products before that
        assert float((out[lo:hi].cpu().double() - y).abs().amax()) <= (3 if glu else 1) * 2.0 ** -8 * max(float(y.abs().amax()), 1e-3)
    assert bool(out[M].isnan().all())
    # the same rows as one group alone, with as many more rows as make the tiles larger
    e = G // 3
    lo, hi = int(off[e]), int(off[e + 1])
    many = torch.cat([rows[lo:hi], rows[:1].expand(60)])
    alone = torch.empty(len(many), N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(a.cuda(), w[e:e + 1].cuda(), alone, group_off=torch.tensor([0, len(many)], dtype=torch.int32, device="cuda"), a_rows=many.cuda(),
                     n_rows=len(many), glu=glu, row_scale=scale.cuda())
    assert torch.equal(alone[:hi - lo], out[lo:hi])


@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33])
def test_batched(cuda_device, M):
    from infinilm_b200 import ops
    G, K, N = 5, 72, 100
    g = torch.Generator().manual_seed(M)
    a, w = torch.randn(M, G, K, generator=g).bfloat16(), (torch.randn(G, N, K, generator=g) * 0.2).bfloat16()
    out = torch.empty(M, G, N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_grouped(a.cuda(), w.cuda(), out)
    ref = torch.einsum("mgk,gnk->mgn", a.double(), w.double())
    assert float((out.cpu().double() - ref).abs().amax()) <= 2.0 ** -8 * float(ref.abs().amax())


@pytest.mark.parametrize("glu", [False, True])
@pytest.mark.parametrize("N,K", [(64, 64), (100, 1408)])
def test_groups_at_the_edges_of_tiles(cuda_device, N, K, glu):
    """A tile of 32 rows with at most 16 leaves its upper half out: groups of 1 to 65 rows together in tiles of 32 (many groups) and of 64 (few), against
    float64 and with the same bits."""
    from infinilm_b200 import ops
    counts = [1, 15, 16, 17, 0, 31, 32, 33, 48, 49, 64, 65, 2]
    M, many = sum(counts), [0] * 20
    g = torch.Generator().manual_seed(N)
    a = torch.randn(M, K, generator=g).bfloat16()
    w = (torch.randn(len(counts), (2 if glu else 1) * N, K, generator=g) * 2 / math.sqrt(K)).bfloat16()
    outs = []
    for pad, rows in ((many, M), ([], M), ([], 64 * M)):           # (n_rows bounds the places and chooses the tile)
        off = torch.tensor([0] + counts + pad).cumsum(0)
        wide = torch.cat([w, w[:1].expand(len(pad), -1, -1)]).contiguous()
        out = torch.full((rows + 1, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        src = torch.cat([a, a[:1].expand(rows - M, -1)]).contiguous()
        ops.gemm_grouped(src.cuda(), wide.cuda(), out[:rows], group_off=off.to(torch.int32).cuda(), n_rows=rows, glu=glu)
        outs.append(out[:M])
        assert bool(out[M:].isnan().all())
        assert torch.equal(outs[-1], outs[0])
    at = 0
    for e, n in enumerate(counts):
        if n:
            y = a[at:at + n].double() @ w[e].double().t()
            if glu:
                gt, up = y[:, :N].bfloat16().double(), y[:, N:].bfloat16().double()
                y = gt * torch.sigmoid(gt) * up
            # rounded to bfloat16 once; with a gate its two products before that
            assert float((outs[0][at:at + n].cpu().double() - y).abs().amax()) <= (3 if glu else 1) * 2.0 ** -8 * float(y.abs().amax())
        at += n


@pytest.mark.parametrize("T", [1, 8, 40])
def test_early_reads_in_a_replayed_chain(cuda_device, T):
    """Layers of sort, gate+up and back product over the same buffers, the back product reading its weights and groups while gate+up still
    runs: replayed as a graph, the bits of the same launches one at a time. (A choice's row is looked up by its place: the sort's atomics order an expert's rows.)"""
    from infinilm_b200 import ops
    E, top, W, F, L = 16, 4, 256, 192, 6
    g = torch.Generator().manual_seed(T)
    choices = [torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32).cuda() for _ in range(L)]
    wgu = [(torch.randn(E, 2 * F, W, generator=g) / W ** 0.5).bfloat16().cuda() for _ in range(L)]
    wd = [(torch.randn(E, W, F, generator=g) / F ** 0.5).bfloat16().cuda() for _ in range(L)]
    x = torch.randn(T, W, generator=g).bfloat16().cuda()
    off, row = torch.empty(E + 1, dtype=torch.int32, device="cuda"), torch.empty(T * top, dtype=torch.int32, device="cuda")
    pos = [torch.empty(T * top, dtype=torch.int32, device="cuda") for _ in range(L)]
    act, y = torch.empty(T * top, F, dtype=torch.bfloat16, device="cuda"), [torch.empty(T * top, W, dtype=torch.bfloat16, device="cuda") for _ in range(L)]

    def run(wait):
        for i in range(L):
            ops.moe_sort(choices[i], E, off, pos[i], row)
            wait()
            ops.gemm_grouped(x, wgu[i], act, group_off=off, a_rows=row, n_rows=T * top, glu=True)
            wait()
            ops.gemm_grouped(act, wd[i], y[i], group_off=off, n_rows=T * top, early=True)
            wait()
    run(torch.cuda.synchronize)
    want = [t[p.long()] for t, p in zip(y, pos)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(lambda: None)
    for _ in range(20):
        for t in y:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(t[p.long()], b) for t, p, b in zip(y, pos, want))
