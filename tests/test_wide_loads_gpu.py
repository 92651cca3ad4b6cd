"""Elementwise kernels that read 16 bytes a thread where sizes and alignment allow it: against float64, and the same bits as the narrow form
gives for the same rows at an odd offset."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def _close(got, ref, dtype):
    assert float((got.double() - ref).abs().amax()) <= (2.0 ** -8 if dtype == "bfloat16" else 2.0 ** -21) * float(ref.abs().amax())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("T,N", [(1, 8), (5, 24), (300, 2560), (70, 2052)])
def test_bias_sum_and_gate(cuda_device, T, N, dtype):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + N)
    a, b, z = (torch.randn(T, N, device="cuda", generator=g).to(DT[dtype]) for _ in range(3))
    bias = torch.randn(N, device="cuda", generator=g)

    def odd(t):                                   # the same rows, not 16-byte aligned
        store = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)
        store[1:] = t.reshape(-1)
        return store[1:].view(t.shape)
    y, y2 = a.clone(), odd(a)
    ops.add_bias(y, bias)
    ops.add_bias(y2, bias)
    _close(y, a.double() + bias.double(), dtype)
    assert torch.equal(y, y2)
    out, out2 = torch.empty_like(a), odd(a)
    ops.scaled_sum(a, 0.5, b, -1.5, out)
    ops.scaled_sum(odd(a), 0.5, odd(b), -1.5, out2)
    _close(out, 0.5 * a.double() - 1.5 * b.double(), dtype)
    assert torch.equal(out, out2)
    y, y2 = a.clone(), odd(a)
    ops.sigmoid_gate(y, z)
    ops.sigmoid_gate(y2, odd(z))
    _close(y, a.double() * torch.sigmoid(z.double()), dtype)
    assert torch.equal(y, y2)


@pytest.mark.parametrize("gate,out_dtype", [("float32", "float32"), ("float32", "bfloat16"), ("bfloat16", "bfloat16")])
@pytest.mark.parametrize("T,group,n_groups", [(3, 516, 2), (300, 2048, 1), (2, 2052, 1), (1, 4096, 1), (5, 4100, 2), (2, 8192, 1), (2, 8196, 1), (4, 2050, 1)])
def test_norms_over_wide_groups(cuda_device, T, group, n_groups, gate, out_dtype):
    from infinilm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + group)
    n = group * n_groups
    x, w = torch.randn(T, n, device="cuda", generator=g) * 3, 1 + 0.1 * torch.randn(n, device="cuda", generator=g)
    z = torch.randn(T, n + 8, device="cuda", generator=g).to(DT[gate])
    for act in (ops.GATE_SIGMOID, ops.GATE_SILU):
        out = torch.full((T, n), float("nan"), device="cuda", dtype=DT[out_dtype])
        ops.group_norm_gate(x, w, 1e-5, z, 4, act, out, group)
        xd, zd = x.double().view(T, n_groups, group), z[:, 4:4 + n].double()
        y = (xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-5)).view(T, n) * w.double()
        ref = y * torch.sigmoid(zd) * (zd if act == ops.GATE_SILU else 1.0)
        _close(out, ref, out_dtype)


@pytest.mark.parametrize("x_dtype,out_dtype", [("float32", "float32"), ("bfloat16", "float32"), ("bfloat16", "bfloat16")])
@pytest.mark.parametrize("C", [4, 520, 2560])
@pytest.mark.parametrize("act", [0, 1])
def test_short_convolution_of_long_portions(cuda_device, C, act, x_dtype, out_dtype):
    """Entries of 1 to 130 tokens in one step of more than 64, from a state and from nothing: four channels a thread and, at an odd column, one."""
    from infinilm_b200 import ops
    lens, taps = [1, 130, 2, 3, 8, 1, 17, 4], 4
    T, E = sum(lens), len(lens)
    g = torch.Generator(device="cuda").manual_seed(C + act)
    qs = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    ent = torch.repeat_interleave(torch.arange(E), torch.tensor(lens)).to(torch.int32).cuda()
    rd = torch.tensor([0, 1, 2, 0, 4, 5, 6, 7], dtype=torch.int32, device="cuda")
    wr = torch.tensor([9, 1, 2, 3, 4, 5, 6, 7], dtype=torch.int32, device="cuda")
    w = torch.randn(C, taps, device="cuda", generator=g)
    state0 = torch.randn(10, taps - 1, C, device="cuda", generator=g)
    state0[0] = 0
    wide = torch.randn(T, C + 8, device="cuda", generator=g).to(DT[x_dtype])
    outs = []
    for off in (4, 3):
        x = torch.empty(T, C + 8, device="cuda", dtype=DT[x_dtype])
        x[:, off:off + C] = wide[:, 4:4 + C]
        state, out = state0.clone(), torch.full((T, C + 8), float("nan"), device="cuda", dtype=DT[out_dtype])
        ops.short_conv(x, off, w, state, 0, rd, ent, qs, out, off, 1, C, C, act, write_slots=wr)
        outs.append((out[:, off:off + C].clone(), state))
        assert bool(out[:, :off].isnan().all()) and bool(out[:, off + C:].isnan().all())
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    xd = wide[:, 4:4 + C].double()
    for e in range(E):
        a, b = int(qs[e]), int(qs[e + 1])
        u = torch.cat([state0[int(rd[e])].double(), xd[a:b]])
        y = sum(w[:, j].double() * u[j:j + b - a] for j in range(taps))
        ref = y * torch.sigmoid(y) if act else y
        _close(outs[0][0][a:b], ref, out_dtype)
        if b - a == 1:
            assert torch.equal(outs[0][1][int(wr[e])], u[1:].float())


@pytest.mark.parametrize("T", [255, 256, 300])
@pytest.mark.parametrize("H,top", [(64, 1), (520, 8), (2048, 6), (2056, 9), (1036, 3)])
@pytest.mark.parametrize("shared,identity", [(True, False), (False, True), (True, True)])
def test_combining_the_rows_of_many_tokens(cuda_device, T, H, top, shared, identity):
    """Few tokens and many, columns in steps of 8 and of 4, one round of choices and more, choices that return the input."""
    from infinilm_b200 import ops
    g = torch.Generator().manual_seed(T + H)
    pos = torch.randperm(T * top, generator=g).to(torch.int32)
    y, x = torch.randn(T * top, H, generator=g).bfloat16(), torch.randn(T, H, generator=g).bfloat16()
    wt = torch.rand(T, top, generator=g)
    sh, sg = torch.randn(T, H, generator=g).bfloat16() if shared else None, torch.randn(T, generator=g) if shared and identity else None
    n_real, cut = 3, T * top * 3 // 4
    off = torch.tensor([0, 5, 9, cut, T * top], dtype=torch.int32)
    out = torch.full((T, H), float("nan"), dtype=torch.bfloat16, device="cuda")
    c = lambda t: None if t is None else t.cuda()
    ops.moe_combine(y.cuda(), pos.cuda(), wt.cuda(), c(sh), out, top=top, group_off=off.cuda() if identity else None, n_real=n_real if identity else 0,
                    x=x.cuda() if identity else None, shared_gate=c(sg))
    p = pos.view(T, top).long()
    rows = y.double()[p]
    if identity:
        rows = torch.where((p >= cut)[:, :, None], x.double()[:, None, :], rows)
    ref = (wt.double()[:, :, None] * rows).sum(1)
    if shared:
        ref = ref + (torch.sigmoid(sg.double())[:, None] if sg is not None else 1.0) * sh.double()
    _close(out.cpu(), ref, "bfloat16")


@pytest.mark.parametrize("T", [3, 300])
def test_choices_of_a_token_end_at_the_room_for_them(cuda_device, T):
    """32 choices are summed, 33 are refused: few tokens and many."""
    from infinilm_b200 import ops
    H = 64
    g = torch.Generator().manual_seed(T)
    for top in (32, 33):
        y, wt = torch.randn(T * top, H, generator=g).bfloat16(), torch.rand(T, top, generator=g)
        pos, out = torch.randperm(T * top, generator=g).to(torch.int32), torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
        if top == 33:
            with pytest.raises(ops.KernelError):
                ops.moe_combine(y.cuda(), pos.cuda(), wt.cuda(), None, out, top=top)
            continue
        ops.moe_combine(y.cuda(), pos.cuda(), wt.cuda(), None, out, top=top)
        _close(out.cpu(), (wt.double()[:, :, None] * y.double()[pos.view(T, top).long()]).sum(1), "bfloat16")
