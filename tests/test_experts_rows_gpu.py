"""The sort of (token, expert) pairs and the sum of a token's expert rows at the edges of their kernels: whole numbers exactly, sums in
the order chosen rounded once (2^-8 of the terms' sizes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,top", [(1, 1, 1), (33, 8, 3), (500, 33, 4), (2048, 32, 4), (700, 256, 8), (40, 300, 2)])
def test_pairs_are_sorted_by_expert_in_their_own_order(T, E, top):
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    offsets, place_of, pair_at = ops.moe_sort(idx.cuda(), E)
    flat = idx.reshape(-1).long()
    order = torch.sort(flat, stable=True).indices
    assert torch.equal(pair_at.cpu().long(), order)
    assert torch.equal(place_of.cpu().long()[order], torch.arange(T * top))
    assert torch.equal(offsets.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat, minlength=E).cumsum(0)]))


@pytest.mark.parametrize("N", [8, 136, 256, 504, 512, 520, 1000, 2048, 2056, 30])
@pytest.mark.parametrize("top,weighted,shared", [(1, False, False), (3, True, True), (4, True, False), (5, False, True), (8, True, True)])
def test_a_tokens_rows_are_summed_in_the_order_chosen(N, top, weighted, shared):
    from tensorline_b200 import ops
    T, E = 37, 9
    g = torch.Generator().manual_seed(N + top)
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32).cuda()
    offsets, place_of, _ = ops.moe_sort(idx, E)
    rows = torch.randn(T * top, N, generator=g).bfloat16().cuda()
    wts = torch.rand(T, top, generator=g).cuda() if weighted else None
    extra = torch.randn(T, N, generator=g).bfloat16().cuda() if shared else None
    gate = torch.randn(T, 3, generator=g).cuda()[:, 1] if shared else None
    y = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    ops.moe_combine(rows, place_of, idx, offsets, wts, y, extra=extra, extra_gate=gate)
    parts = rows.double()[place_of.long().view(T, top)]
    if weighted:
        parts = parts * wts.double()[:, :, None]
    want, size = parts.sum(1), parts.abs().sum(1)
    if shared:
        e = torch.sigmoid(gate.double())[:, None] * extra.double()
        want, size = want + e, size + e.abs()
    assert float(((y.double() - want).abs() - 2.0 ** -8 * want.abs() - 2.0 ** -20 * size).max()) <= 0.0


@pytest.mark.parametrize("adt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,top,K,F,gated", [(1, 1, 8, 3, True), (3, 2, 264, 17, True), (5, 4, 2048, 40, False), (8, 4, 1032, 1, False), (2, 8, 520, 10, True),
                                             (2, 2, 45, 6, True), (3, 2, 64, 256, True), (4, 3, 64, 264, True), (4, 2, 72, 768, False)])
def test_streamed_experts_against_float64_and_token_by_token(T, top, K, F, gated, adt):
    """K products of unit normals with weights of 0.05 in float32, rounded to the activation type (2^-8 for bfloat16)."""
    from tensorline_b200 import ops
    E, real = 9, 8
    g = torch.Generator().manual_seed(T * K + F)
    h = torch.randn(T, K, generator=g).to(adt)
    up = (torch.randn(real, (2 if gated else 1) * F, K, generator=g) * 0.05).bfloat16()
    down = (torch.randn(real, K, F, generator=g) * 0.2).bfloat16()
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    wts = torch.rand(T, top, generator=g)
    act = "silu" if gated else "relu_squared"

    def run(rows):
        n = len(rows)
        a = torch.zeros(n * top, F, dtype=adt, device="cuda")
        y = torch.empty(n, K, dtype=adt, device="cuda")
        hd, ix = h[rows].contiguous().cuda(), idx[rows].contiguous().cuda()
        ops.moe_up(hd, up.cuda(), ix, a, act=act, gated=gated)
        ops.moe_down(a, down.cuda(), ix, wts[rows].contiguous().cuda(), y, same=hd)
        return a, y
    a, y = run(list(range(T)))
    for t in range(T):
        a1, y1 = run([t])
        assert torch.equal(a1, a[t * top:(t + 1) * top]) and torch.equal(y1[0], y[t])
        want, size = torch.zeros(K, dtype=torch.float64), torch.zeros(K, dtype=torch.float64)
        for j in range(top):
            e = int(idx[t, j])
            if e >= real:
                p = h[t].double()
            else:
                u = up[e].double() @ h[t].double()
                u = u[:F] * torch.sigmoid(u[:F]) * u[F:] if gated else torch.relu(u) ** 2
                got = a[t * top + j].double().cpu()
                assert float((got - u).abs().max()) <= (1e-5 if adt == torch.float32 else 2.0 ** -8) * (1 + float(u.abs().max()))
                p = down[e].double() @ got
                size += wts[t, j].double() * (down[e].double().abs() @ got.abs())
            want += wts[t, j].double() * p
            size += (wts[t, j].double() * p).abs()
        rounding = 2.0 ** -8 if adt == torch.bfloat16 else 1e-6
        assert float(((y[t].double().cpu() - want).abs() - rounding * want.abs() - 1e-5 * (1 + size)).max()) <= 0.0
