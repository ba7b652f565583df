"""The float products of few outputs and the per-head norms at the edges of their dispatch.  Bounds: K products of unit normals with
weights of 0.02 in float32 (5e-6 * sqrt(K) is hundreds of roundings); a norm's result rounded once to bfloat16 (2^-9)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,K", [(1, 1, 8), (1, 16, 2048), (32, 33, 2056), (33, 5, 264), (70, 40, 4096), (513, 17, 72), (3, 7, 45), (2100, 33, 512),
                                   (16, 256, 520), (17, 256, 520), (24, 256, 264), (25, 257, 264)])
def test_small_products_at_every_length_of_a_step(T, N, K, adt):
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(T + N + K)
    h, w, b = torch.randn(T, K, generator=g).to(adt).cuda(), (torch.randn(N, K, generator=g) * 0.02).bfloat16().cuda(), torch.randn(N, generator=g).bfloat16().cuda()
    for bias in (None, b):
        out = torch.full((T, N), 7.0, device="cuda")
        ops.small_proj(h, w, bias, out)
        want = h.double() @ w.double().T + (bias.double() if bias is not None else 0.0)
        assert float((out.double() - want).abs().max()) <= 1e-6 + 5e-6 * 0.02 * K ** 0.5
        one = torch.empty(1, N, device="cuda")
        for t in (0, T // 2, T - 1):                     # a token's result does not depend on the others
            ops.small_proj(h[t:t + 1].contiguous(), w, bias, one)
            assert torch.equal(one[0], out[t])


@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16, None])
@pytest.mark.parametrize("T,H,dv,act", [(1, 1, 4, "silu"), (5, 3, 256, "sigmoid"), (2, 5, 132, "silu"), (3, 2, 512, None), (4, 2, 30, "silu"), (2, 2, 520, "sigmoid"),
                                        (3, 5, 60, "silu"), (3, 5, 64, "sigmoid")])
def test_head_norms_against_float64(T, H, dv, act, wdt, gdt):
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(T * dv + H)
    o, gate = torch.randn(T, H * dv, generator=g).cuda(), torch.randn(T, H * dv + 12, generator=g).to(gdt).cuda()
    w = None if wdt is None else torch.randn(H * dv, generator=g).to(wdt).cuda()
    out = torch.empty(T, H * dv, dtype=torch.bfloat16, device="cuda")
    ops.head_norm_gate(o, out, H, dv, 1e-5, weight=w, gate=gate if act else None, gate_off=8, act=act)
    x = o.double().view(T, H, dv)
    want = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).view(T, H * dv)
    if w is not None:
        want = want * w.double()
    if act:
        z = gate[:, 8:8 + H * dv].double()
        want = want * torch.sigmoid(z) * (z if act == "silu" else 1.0)
    assert float(((out.double() - want).abs() - 2.0 ** -8 * want.abs()).max()) <= 1e-6
