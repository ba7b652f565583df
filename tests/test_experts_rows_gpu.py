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


@pytest.mark.parametrize("N", [8, 136, 2048, 2056, 30])
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
