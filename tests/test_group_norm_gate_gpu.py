"""The norm over groups times a gate, a warp a group and a block a group, at the edges between the two."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,n_groups", [(4, 3), (124, 2), (128, 16), (132, 5), (256, 8), (260, 1), (512, 4), (516, 2), (126, 3)])
@pytest.mark.parametrize("T,offset", [(1, 0), (8, 4), (75, 1), (300, 8)])
@pytest.mark.parametrize("gate_dtype,out_dtype", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16)])
def test_against_float64(cuda_device, group, n_groups, T, offset, gate_dtype, out_dtype):
    """offset: columns in front of the gate's (1: its pieces are not aligned, the general kernel takes the call)."""
    from infinilm_b200 import ops
    n = group * n_groups
    g = torch.Generator().manual_seed(group + T)
    x = torch.randn(T, n, generator=g)
    gate = (2 * torch.randn(T, n + offset + (-offset) % 4 + 4, generator=g)).to(gate_dtype)
    for act, n_w, w_dtype in ((0, group, torch.float32), (1, n, torch.bfloat16)):
        w = (1 + 0.2 * torch.randn(n_w, generator=g)).to(w_dtype)
        out = torch.full((T, n + 4), float("nan"), dtype=out_dtype, device="cuda")
        ops.group_norm_gate(x.cuda(), w.cuda(), 1e-5, gate.cuda(), offset, act, out[:, :n], group)
        xg = x.double().view(T, n_groups, group)
        y = (xg * torch.rsqrt((xg * xg).mean(-1, keepdim=True) + 1e-5)).view(T, n) * w.double().repeat(n // n_w)
        z = gate[:, offset:offset + n].double()
        ref = y * (torch.sigmoid(z) if act == 0 else z * torch.sigmoid(z))
        tol = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -19        # one rounding to the type; f32 sums and the unit for exp before it
        assert bool(((out[:, :n].cpu().double() - ref).abs() <= tol * ref.abs() + 1e-7).all())
        assert bool(out[:, n:].isnan().all())


@pytest.mark.parametrize("group", [516, 1020, 1024, 1028, 2044, 2048, 2052, 4096, 4100, 8192])
@pytest.mark.parametrize("gate_dtype,out_dtype,act", [(torch.float32, torch.float32, 0), (torch.bfloat16, torch.bfloat16, 1)])
def test_wide_groups_in_pieces_and_a_column_a_thread(cuda_device, group, gate_dtype, out_dtype, act):
    """Groups of more than 512 columns: the same bits from the kernel of 16-byte pieces and, the gate at an odd column, from that of one column a thread."""
    from infinilm_b200 import ops
    T, n = 5, 2 * group
    g = torch.Generator(device="cuda").manual_seed(group)
    x, w = torch.randn(T, n, device="cuda", generator=g) * 3, torch.randn(n, device="cuda", generator=g)
    z = torch.randn(T, n, device="cuda", generator=g).to(gate_dtype)
    outs = []
    for off in (4, 5):
        gate = torch.zeros(T, n + 8, device="cuda", dtype=gate_dtype)
        gate[:, off:off + n] = z
        out = torch.full((T, n), float("nan"), device="cuda", dtype=out_dtype)
        ops.group_norm_gate(x, w, 1e-5, gate, off, act, out, group)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    xd, zd = x.double().view(T, 2, group), z.double()
    ref = (xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-5)).view(T, n) * w.double() * (torch.sigmoid(zd) if act == 0 else zd * torch.sigmoid(zd))
    # float32: a dozen roundings and two short functions; bfloat16: the result's own
    bound = ref.abs() * (2.0 ** -19 if out_dtype == torch.float32 else 2.0 ** -8) + 1e-30
    assert bool(((outs[0].double() - ref).abs() <= bound).all())
