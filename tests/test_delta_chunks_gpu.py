"""The delta rule in chunks (`ops.delta_chunks`): against the recurrence in float64 over the forms it accepts and beside the
token-by-token kernel, whose state it shares: its error may be no larger than that kernel's, give or take one rounding (2^-24)."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def slot_rows(S):
    H, d, dv = S.shape
    R, IS = (4, 8) if d <= 32 else (8, 8) if d <= 64 else (8, 16) if d <= 128 else (8, 32)
    nz = -(-dv // 16)
    out = torch.zeros(H, nz, R * IS * 16, dtype=S.dtype)
    i, j = torch.meshgrid(torch.arange(d), torch.arange(dv), indexing="ij")
    out[:, j // 16, (i % R) * IS * 16 + (j % 16) * IS + i // R] = S
    return out.reshape(-1)


@pytest.mark.parametrize("H,nqk,d,dv,lens,like", [
    (4, 2, 128, 256, [64, 33, 1], 0.0), (2, 2, 64, 64, [200], 0.0), (3, 1, 36, 132, [31, 32, 97], 0.0), (2, 1, 64, 36, [70], 0.0),
    (2, 2, 40, 20, [40, 3], 0.0), (2, 1, 96, 128, [160], 0.9), (1, 1, 124, 64, [65], 0.0), (1, 1, 128, 4, [129], 0.5), (2, 2, 128, 64, [96], 0.99)])
def test_delta_chunks_against_the_recurrence_in_float64(H, nqk, d, dv, lens, like):
    """`like`: how alike the keys are (the system of a chunk is the further from the identity)."""
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(d * dv + sum(lens))
    T, B = sum(lens), len(lens)
    q, k = torch.randn(T, nqk, d, generator=g), torch.randn(T, nqk, d, generator=g) * (1 - like) + like * torch.randn(1, nqk, d, generator=g)
    q, k = q / q.norm(dim=-1, keepdim=True) * d ** -0.5, k / k.norm(dim=-1, keepdim=True)
    v = torch.randn(T, H, dv, generator=g)
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1)
    gates = torch.randn(T, 2 * H + 4, generator=g)
    gates[T // 2, H:2 * H] = 60.0                        # everything before is forgotten here
    A_log, dt_bias = torch.randn(H, generator=g) - 2.0, torch.randn(H, generator=g) - 1.0
    S0 = torch.randn(B, H, d, dv, generator=g) * 0.3
    q_start = [0]
    for n in lens:
        q_start.append(q_start[-1] + n)
    slots = torch.arange(B, 0, -1, dtype=torch.int32)
    first = torch.stack([torch.zeros_like(slot_rows(S0[0]))] + [slot_rows(S0[b]) for b in range(B)][::-1])
    qs, sl = torch.tensor(q_start, dtype=torch.int32).cuda(), slots.cuda()
    args = (qkv.cuda(), gates.cuda(), A_log.cuda(), dt_bias.cuda())
    state, out = first.cuda(), torch.full((T, H * dv), 7.0, device="cuda")
    ops.delta_chunks(*args, state, SimpleNamespace(h_q_start=q_start, scratch={}, q_start=qs, slots=sl), out, H=H, nqk=nqk, d=d, dv=dv)
    scan_state, scan_out = first.cuda(), torch.empty_like(out)
    ops.delta_scan(*args, scan_state, qs, sl, scan_out, B=B, H=H, nqk=nqk, d=d, dv=dv, max_q_len=max(lens))
    rep = H // nqk
    q64, k64, v64, g64 = (x.double() for x in (q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1), v, gates))
    beta = torch.sigmoid(g64[:, :H])
    decay = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(g64[:, H:2 * H] + dt_bias.double()))
    for b in range(B):
        S, o = S0[b].double(), []
        for t in range(q_start[b], q_start[b + 1]):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v64[t] - torch.einsum("hd,hde->he", k64[t], S))
            S = S + k64[t][:, :, None] * u[:, None, :]
            o.append(torch.einsum("hd,hde->he", q64[t], S).reshape(-1))
        rows = slice(q_start[b], q_start[b + 1])
        for got, scan, want in ((out[rows], scan_out[rows], torch.stack(o)), (state[int(slots[b])], scan_state[int(slots[b])], slot_rows(S))):
            err, base = (float((y.double().cpu() - want).norm()) / float(want.norm()) for y in (got, scan))
            assert err <= 1.05 * base + 2.0 ** -24, (err, base)
    assert torch.equal(state[0].cpu(), first[0])


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("H,d,dv,T", [(8, 128, 256, 300), (4, 128, 128, 130), (8, 96, 64, 300), (16, 64, 128, 200)])
def test_errors_are_no_larger_than_token_by_token(H, d, dv, T, seed):
    """Sizes and distributions as the decoders have them, from a state of zero: the error of outputs and states against 64 bits is no
    larger than the token-by-token kernel's; 1.02: what is left of draws of this size."""
    from tensorline_b200 import ops
    nqk = H // 2
    g = torch.Generator().manual_seed(seed + T)
    q, k, v = torch.randn(T, nqk, d, generator=g), torch.randn(T, nqk, d, generator=g), torch.randn(T, H, dv, generator=g) * 0.5
    q, k = q / q.norm(dim=-1, keepdim=True) * d ** -0.5, k / k.norm(dim=-1, keepdim=True)
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1)
    gates, A_log, dt_bias = torch.randn(T, 2 * H, generator=g) * 0.9, torch.randn(H, generator=g) * 1.2 - 2, torch.randn(H, generator=g) - 1
    floats = H * -(-dv // ops.delta_columns()) * ops.delta_state_floats(d)
    i32 = dict(dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(h_q_start=[0, T], scratch={}, q_start=torch.tensor([0, T], **i32), slots=torch.zeros(1, **i32))
    outs, states = [torch.empty(T, H * dv, device="cuda") for _ in range(2)], [torch.zeros(1, floats, device="cuda") for _ in range(2)]
    args = [x.cuda() for x in (qkv, gates, A_log, dt_bias)]
    ops.delta_chunks(*args, states[0], ctx, outs[0], H=H, nqk=nqk, d=d, dv=dv)
    ops.delta_scan(*args, states[1], ctx.q_start, ctx.slots, outs[1], B=1, H=H, nqk=nqk, d=d, dv=dv, max_q_len=T)
    q64, k64 = (x.double().repeat_interleave(2, 1) for x in (q, k))
    beta = torch.sigmoid(gates[:, :H].double())
    decay = torch.exp(-torch.exp(A_log.double()) * torch.nn.functional.softplus(gates[:, H:].double() + dt_bias.double()))
    S, o = torch.zeros(H, d, dv, dtype=torch.float64), []
    for t in range(T):
        S = decay[t][:, None, None] * S
        S = S + k64[t][:, :, None] * (beta[t][:, None] * (v[t].double() - torch.einsum("hd,hde->he", k64[t], S)))[:, None, :]
        o.append(torch.einsum("hd,hde->he", q64[t], S).reshape(-1))
    for got, want in ((outs, torch.stack(o)), ([s[0] for s in states], slot_rows(S))):
        err, base = (float((y.double().cpu() - want).norm()) / float(want.norm()) for y in got)
        assert err <= 1.02 * base, (err, base)


def test_decays_of_zero_forget_as_token_by_token():
    """Log decays that a float does not hold, or that would swallow their neighbours' in a sum, beside ordinary ones."""
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(9)
    H, nqk, d, dv, T = 3, 3, 64, 64, 100
    qkv = torch.randn(T, H * (2 * d + dv), generator=g) * d ** -0.5
    gates = torch.randn(T, 2 * H, generator=g)
    gates[::7, H:] = 3e37                                # heads 0 and 1: products of 1e38 and more; head 2: every token
    A_log, dt_bias = torch.tensor([3.0, 1.0, 100.0]), torch.zeros(H)
    args = [x.cuda() for x in (qkv, gates, A_log, dt_bias)]
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, False)
    first = torch.randn(2, floats, generator=g).cuda()
    qs, sl = torch.tensor([0, T], dtype=torch.int32).cuda(), torch.tensor([1], dtype=torch.int32).cuda()
    got, want = (torch.empty(T, H * dv, device="cuda") for _ in range(2))
    state, scan_state = first.clone(), first.clone()
    ops.delta_chunks(*args, state, SimpleNamespace(h_q_start=[0, T], scratch={}, q_start=qs, slots=sl), got, H=H, nqk=nqk, d=d, dv=dv)
    ops.delta_scan(*args, scan_state, qs, sl, want, B=1, H=H, nqk=nqk, d=d, dv=dv, max_q_len=T)
    for a, b in ((got, want), (state, scan_state)):
        assert bool(b.isfinite().all()) and float((a - b).norm()) <= 4e-6 * float(b.norm())      # 2e-6 for either kernel, as above


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("k", -float("inf")), ("v", 1e30), ("q", float("nan")),
                                        ("beta", float("nan")), ("decay", float("nan"))])
@pytest.mark.parametrize("d,dv", [(64, 68), (128, 128)])
def test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, d, dv):
    """One element of one token (number 37 of 200) of one of two requests: tokens before it, other heads and the other request are as
    they are without it; with one in the keys, the values or the gates the heads that read it have the token-by-token kernel's floats."""
    from tensorline_b200 import ops
    H, nqk, T, lens = 4, 2, 380, [180, 200]
    g = torch.Generator().manual_seed(d + dv)
    clean = torch.randn(T, 2 * nqk * d + H * dv, generator=g) * d ** -0.5
    gates = torch.randn(T, 2 * H, generator=g)
    odd, odd_gates = clean.clone(), gates.clone()
    at = lens[0] + 37
    if what in ("beta", "decay"):
        odd_gates[at, 2 + (H if what == "decay" else 0)] = value
    else:
        odd[at, {"q": d, "k": nqk * d + d, "v": 2 * nqk * d + 2 * dv}[what] + 3] = value
    hit = [2, 3] if what in "qk" else [2]                # heads 2 and 3 share the second q/k head
    others = [h for h in range(H) if h not in hit]
    floats = H * -(-dv // ops.delta_columns()) * ops.delta_state_floats(d)
    i32 = dict(dtype=torch.int32, device="cuda")
    start = torch.tensor([0, lens[0], T], **i32)
    ctx = SimpleNamespace(h_q_start=start.tolist(), scratch={}, q_start=start, slots=torch.arange(2, **i32))
    consts = (torch.randn(H, generator=g).cuda() - 2.0, torch.randn(H, generator=g).cuda() - 1.0)

    def run(x, gt, chunks):
        state, out = torch.zeros(2, floats, device="cuda"), torch.empty(T, H * dv, device="cuda")
        if chunks:
            ops.delta_chunks(x.cuda(), gt.cuda(), *consts, state, ctx, out, H=H, nqk=nqk, d=d, dv=dv)
        else:
            ops.delta_scan(x.cuda(), gt.cuda(), *consts, state, ctx.q_start, ctx.slots, out, B=2, H=H, nqk=nqk, d=d, dv=dv, max_q_len=200)
        return out.view(T, H, dv), state.view(2, H, -1)
    (out, state), (want, want_state), (fine, fine_state) = run(odd, odd_gates, True), run(odd, odd_gates, False), run(clean, gates, True)
    assert torch.equal(out[:lens[0]], fine[:lens[0]]) and torch.equal(state[0], fine_state[0])
    assert torch.equal(out[:, others], fine[:, others]) and torch.equal(state[1, others], fine_state[1, others])
    if what == "q":
        assert torch.equal(out[lens[0]:at], fine[lens[0]:at]) and torch.equal(out[at + 1:], fine[at + 1:]) and torch.equal(state, fine_state)
        assert bool(out[at, hit].isnan().all())
    else:
        assert bool(want[:at].isfinite().all())
        torch.testing.assert_close(out[lens[0]:, hit], want[lens[0]:, hit], rtol=0, atol=0, equal_nan=True)
        torch.testing.assert_close(state[1, hit], want_state[1, hit], rtol=0, atol=0, equal_nan=True)


def test_short_requests_beside_a_portion_have_the_token_by_token_kernels_floats():
    """Decoding requests and short portions in a step that holds long ones: outputs and states as the scan kernel gives them, whatever
    runs beside them; and the long ones' do not depend on the short ones."""
    from tensorline_b200 import ops
    H, nqk, d, dv, lens, least = 4, 2, 64, 68, [1, 1, 130, 32, 31, 0, 1, 300, 7], 32
    T, B = sum(lens), len(lens)
    g = torch.Generator().manual_seed(d)
    args = [torch.randn(*s, generator=g).cuda() * x for s, x in (((T, 2 * nqk * d + H * dv), d ** -0.5), ((T, 2 * H), 1.0), ((H,), 1.0), ((H,), 1.0))]
    first = torch.randn(B, H * -(-dv // ops.delta_columns()) * ops.delta_state_floats(d), generator=g).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    ctx = SimpleNamespace(h_q_start=start.tolist(), scratch={}, q_start=start, slots=torch.arange(B, **i32).flip(0).contiguous())
    got = []
    for n in (least, 1, None):
        state, out = first.clone(), torch.full((T, H * dv), 7.0, device="cuda")
        if n is None:
            ops.delta_scan(*args, state, start, ctx.slots, out, B=B, H=H, nqk=nqk, d=d, dv=dv, max_q_len=300)
        else:
            ops.delta_chunks(*args, state, ctx, out, H=H, nqk=nqk, d=d, dv=dv, least=n)
        got.append((out, state))
    for b, n in enumerate(lens):
        rows, slot = slice(int(start[b]), int(start[b + 1])), int(ctx.slots[b])
        want, want_state = got[1 if n >= least else 2]
        assert torch.equal(got[0][0][rows], want[rows]) and torch.equal(got[0][1][slot], want_state[slot]), n


def test_heads_that_run_token_by_token_are_refused():
    from tensorline_b200 import ops
    for d, dv in ((32, 64), (132, 64), (64, 30), (62, 64), (64, 1028)):
        x = torch.zeros(128, 2 * d + dv, device="cuda")
        assert not ops.takes_delta_chunks(x, 1, 1, d, dv, 128)
    assert ops.takes_delta_chunks(torch.zeros(128, 192, device="cuda"), 1, 1, 64, 64, 128)
