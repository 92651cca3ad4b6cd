"""The slots' order by expert, and the latent rows' norm, at the sizes where their kernels change form."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 31, 32, 33, 64, 200])
@pytest.mark.parametrize("T,top", [(1, 1), (8, 8), (341, 3), (512, 2), (1025, 1), (700, 6)])
def test_sort_by_expert(cuda_device, E, T, top):
    """Against counting: a block sorts up to 1,024 slots with one read of a choice, more in rounds, from 4,096 in two kernels. A choice that names no
    expert has no place."""
    from infinilm_b200 import ops
    g = torch.Generator().manual_seed(E + T)
    idx = torch.randint(0, E, (T, top), generator=g, dtype=torch.int32)
    if T > 8:
        idx[3, 0] = -1
    off = torch.full((E + 1,), -7, dtype=torch.int32, device="cuda")
    pos, row = torch.full((T * top,), -7, dtype=torch.int32, device="cuda"), torch.full((T * top,), -7, dtype=torch.int32, device="cuda")
    ops.moe_sort(idx.cuda(), E, off, pos, row)
    flat = idx.view(-1).long()
    counts = torch.bincount(flat[flat >= 0], minlength=E)
    assert off.cpu().tolist() == [0] + counts.cumsum(0).tolist()
    pos, row = pos.cpu().long(), row.cpu().long()
    live = flat >= 0
    assert bool((pos[~live] == -1).all())
    assert torch.equal(pos[live].sort().values, torch.arange(int(counts.sum())))
    assert bool(((pos >= off.cpu().long()[flat]) & (pos < off.cpu().long()[flat + 1]))[live].all())
    assert torch.equal(row[pos[live]], (torch.arange(T * top) // top)[live])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("n_a,n_b", [(0, 32), (384, 128), (385, 128), (512, 511), (768, 256), (769, 256), (1536, 512)])
def test_latent_rows(cuda_device, dtype, n_a, n_b, static):
    """Rows that stay in registers (up to four elements a thread) and longer ones, the segments apart from one another."""
    from infinilm_b200 import ops
    T, page = 5, 16
    g = torch.Generator().manual_seed(n_a + n_b)
    proj = torch.randn(T, n_a + n_b + 11, generator=g).to(dtype)
    w_a, w_b = 1 + 0.2 * torch.randn(n_a, generator=g), 1 + 0.2 * torch.randn(n_b, generator=g)
    off_a, off_b = 3, n_a + 7
    pos, ent = torch.tensor([0, 15, 16, 31, 7], dtype=torch.int32), torch.arange(T, dtype=torch.int32)
    bt = torch.randperm(2 * T, generator=g).view(T, 2).to(torch.int32)
    cache = torch.zeros(2 * T, 2, 1, page, n_b, dtype=dtype, device="cuda")
    out_a = torch.empty(T, n_a, dtype=dtype, device="cuda") if n_a else None
    out_b = torch.empty(T, n_b, dtype=dtype, device="cuda")
    wa_dev, wb_dev = w_a.cuda() if n_a else None, w_b.cuda()
    ops.latent_norm_store(proj.cuda(), off_a, n_a, off_b, n_b, wa_dev, wb_dev, 1e-5, out_a, out_b, pos.cuda(), ent.cuda(), bt.cuda(),
                          cache, page, w_static=static)

    def ref(off, n, w):
        x = proj[:, off:off + n].double()
        return x * torch.rsqrt((x * x).mean(1, keepdim=True) + 1e-5) * w.double()
    # one rounding to the type, and f32 sums of up to 1,536 squares and two products before it
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    for got, want in ((out_a, ref(off_a, n_a, w_a) if n_a else None), (out_b, ref(off_b, n_b, w_b))):
        if want is not None:
            assert bool(((got.cpu().double() - want).abs() <= tol * want.abs() + 1e-30).all())
    for t in range(T):
        page_of = int(bt[t, int(pos[t]) // page])
        for plane in (0, 1):
            assert torch.equal(cache[page_of, plane, 0, int(pos[t]) % page], out_b[t])
    assert int((cache != 0).any(-1).sum()) == 2 * T
