"""The 32-bit engine's product and attention at the edges of their dispatch: the same floats whichever kernel a row is given to,
and the formula in float64.  Bounds: a chain of n multiply-adds of unit normals is off by at most n * 2^-24 times the sum of the
absolute products, and in the mean by far less; attention outputs are averages of unit normals."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tensorline_b200 import ops
    return ops


def one_row_at_a_time(ops, a, w, bias):
    out = torch.empty((a.shape[0], w.shape[0]), device="cuda")
    for m in range(a.shape[0]):
        ops.gemm_f32(a[m:m + 1], w, out[m:m + 1], bias)
    return out


@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 33, 16), (4, 9473, 40), (8, 65, 520), (9, 31, 24), (16, 9600, 8), (17, 64, 1032), (32, 100, 72),
                                   (33, 9500, 48), (65, 129, 264), (97, 5000, 40), (130, 20000, 24), (257, 385, 104), (20, 40, 46)])
def test_a_row_of_the_product_has_the_same_floats_in_every_step(ops, M, N, K, wdt):
    g = torch.Generator().manual_seed(M * N + K)
    a = torch.randn(M, K, generator=g).cuda()
    w = torch.randn(N, K, generator=g).to(wdt).cuda()
    bias = torch.randn(N, generator=g).to(wdt).cuda()
    out = torch.full((M, N), 7.0, device="cuda")
    ops.gemm_f32(a, w, out, bias)
    want = a.double() @ w.double().T + bias.double()
    size = a.double().abs() @ w.double().abs().T + 1.0
    assert float(((out.double() - want).abs() / size).max()) <= (K + 1) * 2.0 ** -24
    rows = sorted({0, M // 2, M - 1})
    assert torch.equal(out[rows], one_row_at_a_time(ops, a[rows].contiguous(), w, bias))


@pytest.mark.parametrize("d,g,ps", [(64, 1, 4), (128, 7, 16), (20, 4, 3), (96, 9, 8), (256, 2, 16), (160, 16, 16), (18, 2, 4)])
@pytest.mark.parametrize("option", ["plain", "window", "sink", "chunk"])
def test_attention_rows_have_the_same_floats_in_every_step(ops, d, g, ps, option):
    """Portions and single tokens in one step of more than 64 tokens, the same tokens in short steps, the token-wise kernel, and float64."""
    nkv, scale = 2, d ** -0.5
    nq = nkv * g
    reqs = [(1, 130), (33, 31), (1, 0), (40, 64), (2, 300)]
    gen = torch.Generator().manual_seed(d + g)
    mp = -(-max(n + c for n, c in reqs) // ps)
    pages = len(reqs) * mp
    table = torch.randperm(pages, generator=gen).to(torch.int32).view(len(reqs), mp).contiguous()
    k, v = (torch.randn(pages + 1, nkv, ps, d, generator=gen) for _ in range(2))
    pos = torch.tensor([c + i for n, c in reqs for i in range(n)], dtype=torch.int32)
    slot = torch.tensor([b for b, (n, _) in enumerate(reqs) for _ in range(n)], dtype=torch.int32)
    T = pos.numel()
    q = torch.randn(T, nq * d, generator=gen)
    kw, window = {}, None
    if option == "window":
        window, kw["keep_first"] = 33, 5
    if option == "sink":
        kw["sink"], kw["gate"], kw["cap"] = (torch.randn(nq, generator=gen) * 3).cuda(), torch.randn(T, nq, generator=gen).cuda(), 20.0
    if option == "chunk":
        kw["chunk"], kw["slopes"] = 50, torch.rand(nq, generator=gen).cuda()
    dev = [t.cuda() for t in (q, k, v, table, pos, slot)]

    def run(lo, hi, **hints):
        out = torch.full((hi - lo, nq * d), 7.0, device="cuda")
        part = {n: (x[lo:hi].contiguous() if n == "gate" else x) for n, x in kw.items()}
        qd, kd, vd, td, pd, sd = dev
        ops.attn_tokenwise(qd[lo:hi].contiguous(), nq * d, out, kd, vd, td, ps, pd[lo:hi].contiguous(), sd[lo:hi].contiguous(), nq, nkv, d,
                           window, scale, **part, **hints)
        return out
    whole = run(0, T)
    cuts = [0, 1, 30, 61, T]
    assert torch.equal(whole, torch.cat([run(a, b) for a, b in zip(cuts, cuts[1:])]))
    for hints in (dict(max_ctx=int(pos.max()) + 1), dict(singles=True), dict(max_ctx=int(pos.max()) + 1, singles=True)):
        assert torch.equal(whole, run(0, T, **hints))
    assert torch.equal(whole[34:35], run(34, 35, max_ctx=1))      # position 0
    qd, kd, vd, td, pd, sd = dev
    tokenwise = torch.empty_like(whole)
    ops._check(ops.core().tl_attn_tokenwise(
        ops._ptr(qd), nq * d, ops._ptr(tokenwise), ops.dtype_code(qd.dtype), ops._ptr(kd), ops._ptr(vd), ops._ptr(td), mp, ps, ops._ptr(pd), ops._ptr(sd),
        T, nq, nkv, d, window or 0, scale, ops._ptr(kw.get("sink")), kw.get("keep_first", 0), ops._ptr(kw.get("gate")), kw.get("chunk", 0),
        ops._ptr(kw.get("slopes")), kw.get("cap", 0.0), td.shape[0], kd.shape[0], ops.fault_words(qd.device), ops._stream()), "attn_tokenwise")
    assert torch.equal(whole, tokenwise)
    for t in (0, 1, 33, 34, 74, T - 1):
        p, tab = int(pos[t]), table[int(slot[t])]
        j = torch.arange(p + 1)
        keep = torch.ones(p + 1, dtype=torch.bool)
        if window:
            keep = (j > p - window) | (j < 5)
        if option == "chunk":
            keep = j >= p // 50 * 50
        j = j[keep]
        kk, vv = (x[tab[j // ps].long(), :, j % ps].double() for x in (k, v))
        for h in range(nq):
            s = kk[:, h // g] @ q[t, h * d:(h + 1) * d].double() * scale
            if option == "sink":
                s = 20.0 * torch.tanh(s / 20.0)
                e = torch.cat([s, kw["sink"][h].double().cpu().view(1)])
                w = torch.softmax(e, 0)[:-1] * torch.sigmoid(kw["gate"][t, h].double().cpu())
            else:
                if option == "chunk":
                    s = s - kw["slopes"][h].double().cpu() * (p - j)
                w = torch.softmax(s, 0)
            want = w @ vv[:, h // g]
            assert float((whole[t, h * d:(h + 1) * d].double().cpu() - want).abs().max()) <= 2e-5


@pytest.mark.parametrize("window", [None, 700])
def test_dot_products_of_tables_longer_than_a_grid(ops, window):
    """Few tokens whose table holds more groups of keys than blocks fill the GPU: the same floats as with the table cut to the contexts,
    and as the token-wise kernel."""
    nq, nkv, d, ps, mp = 2, 2, 64, 16, 330
    gen = torch.Generator().manual_seed(1)
    table = torch.randperm(2 * mp, generator=gen).to(torch.int32).view(2, mp).contiguous().cuda()
    k, v = (torch.randn(2 * mp + 1, nkv, ps, d, generator=gen).cuda() for _ in range(2))
    pos = torch.cat([torch.arange(5000, 5060), torch.arange(3, 7)]).to(torch.int32).cuda()
    slot = torch.tensor([0] * 60 + [1] * 4, dtype=torch.int32).cuda()
    q, outs = torch.randn(64, nq * d, generator=gen).cuda(), []
    for hints in ({}, dict(max_ctx=5060), dict(max_ctx=5060, singles=True)):
        outs.append(torch.full((64, nq * d), 7.0, device="cuda"))
        ops.attn_tokenwise(q, nq * d, outs[-1], k, v, table, ps, pos, slot, nq, nkv, d, window, 0.125, **hints)
    outs.append(torch.empty_like(q))
    ops._check(ops.core().tl_attn_tokenwise(
        ops._ptr(q), nq * d, ops._ptr(outs[-1]), ops.dtype_code(q.dtype), ops._ptr(k), ops._ptr(v), ops._ptr(table), mp, ps, ops._ptr(pos), ops._ptr(slot),
        64, nq, nkv, d, window or 0, 0.125, None, 0, None, 0, None, 0.0, 2, k.shape[0], ops.fault_words(q.device), ops._stream()), "attn_tokenwise")
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("nq,nkv,d,T", [(16, 8, 64, 1900), (32, 16, 20, 950), (40, 1, 64, 600), (16, 8, 128, 1900), (16, 16, 64, 950), (16, 16, 128, 950)])
def test_prompts_in_blocks_of_either_size_have_the_token_wise_kernels_floats(ops, nq, nkv, d, T):
    """Three blocks of 64 rows an SM and more, several query heads a KV head and one; two requests, the second on cached tokens."""
    gen = torch.Generator().manual_seed(d + T)
    ps, lens, cached = 16, [T - 70, 70], [0, 50]
    mp = -(-T // ps)
    table = torch.randperm(2 * mp, generator=gen).to(torch.int32).view(2, mp).cuda()
    k, v = (torch.randn(2 * mp, nkv, ps, d, generator=gen).cuda() for _ in range(2))
    pos = torch.tensor([c + i for n, c in zip(lens, cached) for i in range(n)], dtype=torch.int32).cuda()
    slot = torch.tensor([b for b, n in enumerate(lens) for _ in range(n)], dtype=torch.int32).cuda()
    q, out = torch.randn(T, nq * d, generator=gen).cuda(), torch.full((T, nq * d), 7.0, device="cuda")
    ops.attn_tokenwise(q, nq * d, out, k, v, table, ps, pos, slot, nq, nkv, d, None, d ** -0.5)
    want = torch.empty_like(out)
    ops._check(ops.core().tl_attn_tokenwise(
        ops._ptr(q), nq * d, ops._ptr(want), ops.dtype_code(q.dtype), ops._ptr(k), ops._ptr(v), ops._ptr(table), mp, ps, ops._ptr(pos), ops._ptr(slot), T, nq, nkv, d,
        0, d ** -0.5, None, 0, None, 0, None, 0.0, 2, 2 * mp, ops.fault_words(q.device), ops._stream()), "attn_tokenwise")
    assert torch.equal(out, want)
