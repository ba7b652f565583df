"""Matrix memories in chunks (`ops.linear_chunks`): against the recurrence in float64 over the forms it accepts, and against the
token-by-token kernel, whose state it shares.  Bounds: sums of up to a few hundred float products of order one, 2e-5 of the largest, and
in the norm no further off than the token-by-token kernel, give or take one rounding (2^-24; of the running maximum, whose rounding scales a gated state).  A gated output is divided by n . q, which may nearly cancel: what both
kernels can be off by is the roundings of its terms over it, 32 of them (2e-6) times sum |terms| / |n . q| of the output and
of the values it weighs (the norm then says little more than how one token's roundings fell)."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def slot_rows(S, n, m):
    """S [H, d, dv] (n [H, d], m [H]) in the scan kernel's slot layout."""
    H, d, dv = S.shape
    R, IS = (4, 8) if d <= 32 else (8, 8) if d <= 64 else (8, 16) if d <= 128 else (8, 32)
    nz, cols = -(-dv // 16), 16 if n is None else 17
    NT = -(-IS * cols // 32) * 32
    out = torch.zeros(H, nz, R * NT + (4 if n is not None else 0), dtype=S.dtype)
    i, j = torch.meshgrid(torch.arange(d), torch.arange(dv), indexing="ij")
    out[:, j // 16, (i % R) * NT + (j % 16) * IS + i // R] = S
    if n is not None:
        i = torch.arange(d)
        out[:, :, (i % R) * NT + 16 * IS + i // R] = n[:, None, :]
        out[:, :, R * NT] = m[:, None]
    return out.reshape(-1)


def recurrence(x, gates, decay, H, d, dv, S, n, m, pos, inv_freq, rot, interleaved, cap, q_scale, k_scale, den_eps):
    T = x.shape[0]
    q, k, v = x[:, :H * d].view(T, H, d), x[:, H * d:2 * H * d].view(T, H, d), x[:, 2 * H * d:2 * H * d + H * dv].view(T, H, dv)
    if rot:
        a = pos.double()[:, None] * inv_freq.double()
        c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]

        def turn(y):
            y = y.clone()
            e1, e2 = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
            y1, y2 = y[..., e1].clone(), y[..., e2].clone()
            y[..., e1], y[..., e2] = y1 * c - y2 * s, y2 * c + y1 * s
            return y
        q, k = turn(q), turn(k)
    q, k = q * q_scale, k * k_scale
    o = torch.empty(T, H, dv, dtype=torch.float64)
    terms = torch.zeros(T, H, dtype=torch.float64)       # gated: sum |terms of n . q| / |what is divided by|
    size = n.abs() if n is not None else None
    for t in range(T):
        if decay is not None:
            S = decay.double()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            o[t] = torch.einsum("hd,hde->he", q[t], S)
            continue
        li = cap * torch.tanh(gates[t, :H] / cap)
        lf = torch.nn.functional.logsigmoid(cap * torch.tanh(gates[t, H:] / cap))
        new = torch.maximum(lf + m, li)
        a, b = torch.exp(lf + m - new), torch.exp(li - new)
        m = new
        S = a[:, None, None] * S + b[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
        n = a[:, None] * n + b[:, None] * k[t]
        size = a[:, None] * size + b[:, None] * k[t].abs()
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + den_eps
        terms[t] = (size * q[t].abs()).sum(-1) / den
        o[t] = torch.einsum("hd,hde->he", q[t], S) / den[:, None]
    return o.reshape(T, H * dv), S, n, m, terms


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("H,d,dv,lens,rot,interleaved", [
    (3, 128, 256, [64, 65, 1], 64, False), (2, 64, 64, [200], 64, True), (1, 32, 128, [127, 63, 128], 0, False), (2, 256, 128, [130], 256, False),
    (2, 20, 36, [70, 3], 8, True), (1, 96, 20, [300, 64], 96, False), (2, 200, 132, [100], 0, False), (1, 4, 4, [193], 0, False),
    (2, 52, 132, [77, 128], 0, False), (3, 20, 20, [70], 12, False), (3, 20, 20, [70], 6, True), (3, 20, 20, [70], 12, True),
    (2, 20, 20, [5, 4161], 8, False)])                   # more chunks than the carry holds factors of at a time
def test_chunks_against_the_recurrence_in_float64_and_the_scan_kernel(gated, H, d, dv, lens, rot, interleaved):
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(d * dv + sum(lens))
    T, B = sum(lens), len(lens)
    width = 2 * H * d + H * dv + 12
    proj = torch.randn(T, width, generator=g)
    rot = 0 if gated else rot
    gates = torch.cat([torch.randn(T, H, generator=g) * 2 - 1, torch.randn(T, H, generator=g) * 2 + 3], dim=1) if gated else None
    if gated:
        gates[T // 2] = torch.tensor([30.0] * H + [-40.0] * H)      # everything before is forgotten here
    decay = None if gated else 1.0 - 2.0 ** (-1 - 5.0 * torch.arange(H))
    inv = 10000.0 ** (-torch.arange(0, rot, 2).float() / max(rot, 1)) if rot else None
    kw = dict(cap=15.0, q_scale=d ** -0.5, k_scale=1.0, den_eps=1e-6) if gated else dict(k_scale=d ** -0.5, q_scale=1.0)
    q_start = [0]
    for n in lens:
        q_start.append(q_start[-1] + n)
    starts = [17 * b for b in range(B)]
    pos = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, lens)]).to(torch.int32)
    slots = torch.arange(B, 0, -1, dtype=torch.int32)
    S0 = torch.randn(B, H, d, dv, generator=g) * 0.3
    n0 = torch.randn(B, H, d, generator=g) * 0.3 if gated else [None] * B
    m0 = torch.randn(B, H, generator=g) if gated else [None] * B
    first = torch.stack([torch.zeros_like(slot_rows(S0[0], n0[0], m0[0]))] + [slot_rows(S0[b], n0[b], m0[b]) for b in range(B)][::-1])
    dev = {k: v.cuda() for k, v in dict(proj=proj, pos=pos, slots=slots, q=torch.tensor(q_start, dtype=torch.int32)).items()}
    if decay is not None:
        kw.update(decay=decay.cuda())
    if gates is not None:
        kw.update(gates=gates.cuda())
    if rot:
        kw.update(inv_freq=inv.cuda(), rot=rot, pairing="interleaved" if interleaved else "half")
    ctx = SimpleNamespace(h_q_start=q_start, scratch={}, pos=dev["pos"], q_start=dev["q"], slots=dev["slots"])
    state, out = first.cuda(), torch.full((T, H * dv), 7.0, device="cuda")
    ops.linear_chunks(dev["proj"], 0, H * d, 2 * H * d, H, d, dv, state, ctx, out, **kw)
    scan_state, scan_out = first.cuda(), torch.empty_like(out)
    ops.linear_scan(dev["proj"], 0, H * d, 2 * H * d, H, d, dv, scan_state, dev["q"], dev["slots"], dev["pos"], scan_out, B=B, **kw)
    for b in range(B):
        rows = slice(q_start[b], q_start[b + 1])
        o, S, n, m, terms = recurrence(proj[rows].double(), gates[rows].double() if gated else None, decay, H, d, dv, S0[b].double(),
                                n0[b].double() if gated else None, m0[b].double() if gated else None, pos[rows], inv, rot, interleaved,
                                kw.get("cap"), kw["q_scale"], kw["k_scale"], kw.get("den_eps", 0.0))
        want = slot_rows(S, n, m)
        for got, scan, x in ((out[rows], scan_out[rows], o), (state[int(slots[b])], scan_state[int(slots[b])], want)):
            if gated and x is o:
                far = (got.double().cpu() - o).abs().view(-1, H, dv) - 2e-6 * terms[:, :, None] * (o.abs().view(-1, H, dv) + float(proj.abs().max()))
                assert float(far.max()) <= 0.0, float(far.max())
                continue
            err, base = (float((y.double().cpu() - x).norm()) / float(x.norm()) for y in (got, scan))
            rounding = 2.0 ** -24 * (max(1.0, float(m.abs().max())) if gated else 1.0)
            assert err <= 1.05 * base + rounding, (err, base)
            assert float((got.double().cpu() - x).abs().max()) <= max(2e-5 * float(x.abs().max()), 4 * float((scan.double().cpu() - x).abs().max()))
    assert torch.equal(state[0].cpu(), first[0])


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("gated,H,d,dv,T", [(True, 4, 256, 256, 300), (True, 4, 32, 64, 500), (True, 8, 128, 256, 300), (True, 16, 64, 128, 200),
                                            (False, 4, 128, 128, 130), (False, 4, 256, 128, 200), (False, 8, 96, 64, 300)])
def test_errors_are_no_larger_than_token_by_token(gated, H, d, dv, T, seed):
    """Sizes and distributions as the decoders have them, from a state of zero: the error against 64 bits of outputs and states (a
    gated state with its maximum) is no larger than the token-by-token kernel's; 1.02: what is left of draws of this size."""
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(seed + T)
    proj = torch.randn(T, 2 * H * d + H * dv, generator=g) * 0.9
    gates = torch.cat([torch.randn(T, H, generator=g) * 1.3 - 2, torch.randn(T, H, generator=g) * 1.3 + 3], dim=1) if gated else None
    decay = None if gated else torch.tensor([1.0 - 2.0 ** (-5 - 5 * i / (H - 1)) for i in range(H)])
    rot, inv = (0, None) if gated else (d, (1e6 ** (-torch.arange(0, d, 2, dtype=torch.float64) / d)).float())
    scales = dict(q_scale=d ** -0.5, k_scale=1.0) if gated else dict(q_scale=1.0, k_scale=d ** -0.5)
    kw = dict(gates=gates.cuda(), cap=15.0, den_eps=1e-6, **scales) if gated else dict(decay=decay.cuda(), inv_freq=inv.cuda(), rot=rot, **scales)
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, gated)
    i32 = dict(dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(h_q_start=[0, T], scratch={}, pos=torch.arange(T, **i32), q_start=torch.tensor([0, T], **i32), slots=torch.zeros(1, **i32))
    outs, states = [torch.empty(T, H * dv, device="cuda") for _ in range(2)], [torch.zeros(1, floats, device="cuda") for _ in range(2)]
    x = proj.cuda()
    ops.linear_chunks(x, 0, H * d, 2 * H * d, H, d, dv, states[0], ctx, outs[0], **kw)
    ops.linear_scan(x, 0, H * d, 2 * H * d, H, d, dv, states[1], ctx.q_start, ctx.slots, ctx.pos, outs[1], B=1, **kw)
    zero = torch.zeros(H, d, dv, dtype=torch.float64)
    o, S, n, m, _ = recurrence(proj.double(), gates.double() if gated else None, decay, H, d, dv, zero, zero[:, :, 0] if gated else None,
                               zero[:, 0, 0] if gated else None, torch.arange(T), inv, rot, False, 15.0, scales["q_scale"], scales["k_scale"], 1e-6)
    for got, want in ((outs, o), ([s[0] for s in states], slot_rows(S, n, m))):
        err, base = (float((y.double().cpu() - want).norm()) / float(want.norm()) for y in got)
        assert err <= 1.02 * base + (2.0 ** -24 * float(m.abs().max()) if gated and want is not o else 0.0), (err, base)


@pytest.mark.parametrize("decay", [[0.0, 0.9], [-0.5, 0.9], [1e-38, 0.9]])
def test_retention_with_decays_that_have_no_logarithm(decay):
    """They run token by token; a tiny positive one in chunks: each must give what the scan kernel gives, which is the same
    floats for the former, and sums in another order for the latter (2e-6 a kernel)."""
    from tensorline_b200 import ops
    from tensorline_b200.parts import Runtime
    from tensorline_b200.parts.recurrent import Retention
    H, d, dv, T = 2, 64, 64, 200
    part = Retention(Runtime(torch.device("cuda"), torch.bfloat16, 16), 64, H, d, dv, decay, 1e-5)
    g = torch.Generator().manual_seed(3)
    proj = torch.randn(T, 2 * H * d + 2 * H * dv, generator=g).cuda()
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, False)
    first = torch.zeros(2, floats, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(h_q_start=[0, T], scratch={}, decode_only=False, max_q_len=T, B=1, pos=torch.arange(T, **i32), q_start=torch.tensor([0, T], **i32),
                          slots=torch.tensor([1], **i32))
    got, want = (torch.empty(T, H * dv, device="cuda") for _ in range(2))
    state, scan_state = first.clone(), first.clone()
    part._scan(torch.empty(T, 64, dtype=torch.bfloat16, device="cuda"), proj, ctx, state, got)
    ops.linear_scan(proj, 0, H * d, 2 * H * d, H, d, dv, scan_state, ctx.q_start, ctx.slots, ctx.pos, want, B=1, decay=torch.tensor(decay).cuda(),
                    k_scale=d ** -0.5)
    for a, b in ((got, want), (state, scan_state)):
        if min(decay) <= 0.0:
            assert torch.equal(a, b)
        assert bool(b.isfinite().all()) and float((a - b).norm()) <= 4e-6 * float(b.norm())


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("v", float("inf")), ("k", float("nan")), ("k", -float("inf")), ("k", 1e30), ("q", float("nan")),
                                        ("i", float("nan")), ("f", float("nan"))])
@pytest.mark.parametrize("gated,d,dv", [(True, 64, 64), (False, 128, 132), (True, 256, 64), (False, 20, 20)])
def test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, gated, d, dv):
    """One element of one token (number 37 of 200) of head 1 of one of two requests: tokens before it, other heads and the other request
    are as they are without it; with one in the keys, the values or the gates the head has the token-by-token kernel's floats."""
    from tensorline_b200 import ops
    if what in "if" and not gated:
        return
    H, T, lens = 3, 380, [180, 200]
    g = torch.Generator().manual_seed(d + dv)
    clean = torch.randn(T, 2 * H * d + H * dv, generator=g)
    gates = torch.randn(T, 2 * H, generator=g) + 1.0
    odd, odd_gates = clean.clone(), gates.clone()
    at, h = lens[0] + 37, 1
    if what == "i" or what == "f":
        odd_gates[at, h + (H if what == "f" else 0)] = value
    else:
        odd[at, {"q": 0, "k": H * d, "v": 2 * H * d}[what] + h * (dv if what == "v" else d) + 3] = value
    kw = dict(q_scale=d ** -0.5, den_eps=1e-6, cap=15.0) if gated else dict(decay=torch.tensor([0.9, 0.97, 0.99]).cuda(), k_scale=d ** -0.5)
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, gated)
    i32 = dict(dtype=torch.int32, device="cuda")
    start = torch.tensor([0, lens[0], T], **i32)
    ctx = SimpleNamespace(h_q_start=start.tolist(), scratch={}, pos=torch.arange(T, **i32), q_start=start, slots=torch.arange(2, **i32))

    def run(x, gt, chunks):
        state, out, extra = torch.zeros(2, floats, device="cuda"), torch.empty(T, H * dv, device="cuda"), dict(gates=gt.cuda()) if gated else {}
        if chunks:
            ops.linear_chunks(x.cuda(), 0, H * d, 2 * H * d, H, d, dv, state, ctx, out, **kw, **extra)
        else:
            ops.linear_scan(x.cuda(), 0, H * d, 2 * H * d, H, d, dv, state, ctx.q_start, ctx.slots, ctx.pos, out, B=2, **kw, **extra)
        return out.view(T, H, dv), state.view(2, H, -1)
    (out, state), (want, want_state), (fine, fine_state) = run(odd, odd_gates, True), run(odd, odd_gates, False), run(clean, gates, True)
    others = [0, 2]
    assert torch.equal(out[:lens[0]], fine[:lens[0]]) and torch.equal(state[0], fine_state[0])
    assert torch.equal(out[:, others], fine[:, others]) and torch.equal(state[1, others], fine_state[1, others])
    if what == "q":
        assert torch.equal(out[lens[0]:at], fine[lens[0]:at]) and torch.equal(out[at + 1:], fine[at + 1:]) and torch.equal(state, fine_state)
        assert bool(out[at, h].isnan().all())
    else:
        assert bool(want[:at].isfinite().all()) and torch.equal(out[:at, h][lens[0]:], want[:at, h][lens[0]:])
        torch.testing.assert_close(out[lens[0]:, h], want[lens[0]:, h], rtol=0, atol=0, equal_nan=True)
        torch.testing.assert_close(state[1, h], want_state[1, h], rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("gated,d,dv", [(True, 64, 64), (False, 128, 256), (False, 32, 20)])
def test_short_requests_beside_a_portion_have_the_token_by_token_kernels_floats(gated, d, dv):
    """Decoding requests and short portions in a step that holds long ones: outputs and states as the scan kernel gives them, whatever
    runs beside them; and the long ones' do not depend on the short ones."""
    from tensorline_b200 import ops
    H, lens, least = 2, [1, 1, 130, 16, 15, 0, 1, 300, 7], 16
    T, B = sum(lens), len(lens)
    g = torch.Generator().manual_seed(d)
    proj, gates = torch.randn(T, 2 * H * d + H * dv, generator=g).cuda(), torch.randn(T, 2 * H, generator=g).cuda() + 1.0
    kw = dict(gates=gates, q_scale=d ** -0.5, den_eps=1e-6, cap=15.0) if gated else dict(decay=torch.tensor([0.9, 0.99]).cuda(), k_scale=d ** -0.5)
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, gated)
    first = torch.randn(B, floats, generator=g).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    start = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32)
    ctx = SimpleNamespace(h_q_start=start.tolist(), scratch={}, pos=torch.arange(T, **i32), q_start=start, slots=torch.arange(B, **i32).flip(0).contiguous())
    got = []
    for n in (least, 1, None):
        state, out = first.clone(), torch.full((T, H * dv), 7.0, device="cuda")
        if n is None:
            ops.linear_scan(proj, 0, H * d, 2 * H * d, H, d, dv, state, start, ctx.slots, ctx.pos, out, B=B, **kw)
        else:
            ops.linear_chunks(proj, 0, H * d, 2 * H * d, H, d, dv, state, ctx, out, least=n, **kw)
        got.append((out, state))
    for b, n in enumerate(lens):
        rows, slot = slice(int(start[b]), int(start[b + 1])), int(ctx.slots[b])
        want, want_state = got[1 if n >= least else 2]
        assert torch.equal(got[0][0][rows], want[rows]) and torch.equal(got[0][1][slot], want_state[slot]), n
