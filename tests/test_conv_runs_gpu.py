"""The short convolution of the delta rule on steps large enough for runs of tokens a warp: the same bits as every request in steps of
its own, and as steps too short for runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adt,wdt", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("d,dv,lens", [(128, 256, [1100, 1, 500, 3]), (96, 200, [1, 2, 1900]), (128, 192, [1] * 48 + [464]), (256, 36, [700] * 4)])
def test_runs_give_the_bits_of_short_steps(d, dv, lens, taps, adt, wdt):
    from tensorline_b200 import ops
    nqk, nv, T, B = 2, 4, sum(lens), len(lens)
    C = 2 * nqk * d + nv * dv
    g = torch.Generator().manual_seed(d + taps)
    proj, w = torch.randn(T, C + 8, generator=g).to(adt).cuda(), torch.randn(C, taps, generator=g).to(wdt).cuda()
    first = torch.randn(B, taps - 1, C, generator=g).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    start = [0] + torch.tensor(lens).cumsum(0).tolist()
    kw = dict(nqk=nqk, d=d, nv=nv, dv=dv, unit_eps=1e-6, q_scale=d ** -0.5)
    state, out = first.clone(), torch.full((T, C), 7.0, device="cuda")
    ops.conv_prep(proj, w, state, torch.tensor(start, **i32), torch.arange(B, **i32), out, B=B, max_q_len=max(lens), **kw)
    want_state, want = first.clone(), torch.full((T, C), 7.0, device="cuda")
    for b, n in enumerate(lens):
        for a in range(start[b], start[b + 1], 300):
            e = min(a + 300, start[b + 1])
            part = torch.empty(e - a, C, device="cuda")
            ops.conv_prep(proj[a:e], w, want_state, torch.tensor([0, e - a], **i32), torch.tensor([b], **i32), part, B=1, max_q_len=e - a, **kw)
            want[a:e] = part
    assert torch.equal(out, want) and torch.equal(state, want_state)


@pytest.mark.parametrize("taps", [2, 4])
@pytest.mark.parametrize("lens", [[16], [1, 17, 3, 33], [1700, 5], [1] * 40 + [31]])
def test_runs_of_either_length_give_the_bits_of_steps_below_16_tokens(lens, taps):
    """Runs of 4 (few warps) and of 8 tokens, with remainders, against the kernel that takes steps of fewer than 16 tokens."""
    from tensorline_b200 import ops
    nqk, d, nv, dv, B = 2, 64, 6, 96, len(lens)
    C = 2 * nqk * d + nv * dv
    g = torch.Generator().manual_seed(len(lens) + taps)
    proj, w = torch.randn(sum(lens), C, generator=g).cuda(), torch.randn(C, taps, generator=g).bfloat16().cuda()
    first = torch.randn(B, taps - 1, C, generator=g).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    start = [0] + torch.tensor(lens).cumsum(0).tolist()
    kw = dict(nqk=nqk, d=d, nv=nv, dv=dv, unit_eps=1e-6, q_scale=0.125)
    state, out = first.clone(), torch.full((start[-1], C), 7.0, device="cuda")
    ops.conv_prep(proj, w, state, torch.tensor(start, **i32), torch.arange(B, **i32), out, B=B, max_q_len=max(lens), **kw)
    want_state, want = first.clone(), torch.empty(start[-1], C, device="cuda")
    for b in range(B):
        for a in range(start[b], start[b + 1], 15):
            e = min(a + 15, start[b + 1])
            ops.conv_prep(proj[a:e], w, want_state, torch.tensor([0, e - a], **i32), torch.tensor([b], **i32), want[a:e], B=1, max_q_len=e - a, **kw)
    assert torch.equal(out, want) and torch.equal(state, want_state)
