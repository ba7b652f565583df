"""Matrix memories in chunks of 128 tokens (33 to 128 rows a head): what chunks of 64 are asked for, at the edges of the longer ones.  The bounds
are those of the tests they are called from."""
from types import SimpleNamespace

import pytest
import torch

from tests import test_linear_chunks_gpu as chunks

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def wide(monkeypatch):
    from tensorline_b200 import ops
    monkeypatch.setattr(ops, "WIDE_CHUNKS_BLOCKS", {False: 0, True: 0})
    monkeypatch.setattr(ops, "WIDE_CHUNKS_SHARE", 1.0)
    monkeypatch.setattr(ops, "_wide_fills", lambda *a: True)
    yield
    ops.check_device_status()


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("H,d,dv,lens,rot,interleaved", [
    (3, 128, 256, [128, 129, 1], 64, False), (2, 64, 64, [300], 64, True), (1, 36, 128, [127, 63, 256], 0, False), (1, 96, 20, [400, 32], 96, False),
    (2, 68, 388, [160, 257], 8, True), (2, 52, 132, [33, 96], 0, False), (40, 128, 512, [513], 0, False)])
def test_wide_chunks_against_the_recurrence_in_float64_and_the_scan_kernel(gated, H, d, dv, lens, rot, interleaved):
    chunks.test_chunks_against_the_recurrence_in_float64_and_the_scan_kernel(gated, H, d, dv, lens, rot, interleaved)


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("gated,H,d,dv,T", [(True, 8, 128, 256, 300), (True, 16, 64, 128, 200), (False, 4, 128, 128, 130), (False, 8, 96, 64, 300),
                                            (True, 8, 128, 256, 1000)])
def test_errors_are_no_larger_than_token_by_token(gated, H, d, dv, T, seed):
    chunks.test_errors_are_no_larger_than_token_by_token(gated, H, d, dv, T, seed)


@pytest.mark.parametrize("what,value", [("v", float("nan")), ("k", -float("inf")), ("k", 1e30), ("q", float("nan"))])
@pytest.mark.parametrize("gated,d,dv", [(True, 64, 64), (False, 128, 132), (True, 128, 256)])
def test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, gated, d, dv):
    chunks.test_a_value_that_is_no_number_reaches_what_it_reaches_token_by_token(what, value, gated, d, dv)


def both(proj, H, d, dv, gates=None, decay=None, q_scale=1.0):
    """Outputs and states in wide chunks and token by token, one request from a state of zero."""
    from tensorline_b200 import ops
    T, gated = proj.shape[0], gates is not None
    kw = dict(gates=gates.cuda(), cap=15.0, den_eps=1e-6) if gated else dict(decay=decay.cuda())
    floats = H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, gated)
    i32 = dict(dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(h_q_start=[0, T], scratch={}, pos=torch.arange(T, **i32), q_start=torch.tensor([0, T], **i32), slots=torch.zeros(1, **i32))
    got = []
    for chunks in (True, False):
        out, state, x = torch.empty(T, H * dv, device="cuda"), torch.zeros(1, floats, device="cuda"), proj.cuda()
        if chunks:
            ops.linear_chunks(x, 0, H * d, 2 * H * d, H, d, dv, state, ctx, out, q_scale=q_scale, **kw)
        else:
            ops.linear_scan(x, 0, H * d, 2 * H * d, H, d, dv, state, ctx.q_start, ctx.slots, ctx.pos, out, B=1, q_scale=q_scale, **kw)
        got.append((out.view(T, H, dv), state))
    return got


@pytest.mark.parametrize("later", [1, 20, 60])
@pytest.mark.parametrize("gated,d,dv", [(True, 64, 64), (False, 64, 132), (True, 128, 256), (False, 128, 64)])
def test_a_query_whose_product_with_a_later_key_overflows(gated, d, dv, later):
    """A large query, not marked as an operand that chunks can't take; the key that overflows with it is `later` tokens behind, so
    the output is finite.  Bound: float sums of d products and 41 tokens, of values whose sums don't cancel (all are positive)."""
    H, T, at = 2, 200, 40
    g = torch.Generator().manual_seed(later + d)
    proj = torch.rand(T, 2 * H * d + H * dv, generator=g) + 0.5
    proj[at, d:2 * d] = 1e30
    proj[at + later, H * d + d:H * d + 2 * d] = 1e10
    gates = torch.cat([torch.randn(T, H, generator=g), torch.randn(T, H, generator=g) + 3.0], dim=1) if gated else None
    (out, _), (want, _) = both(proj, H, d, dv, gates, None if gated else torch.tensor([0.9, 0.99]))
    assert bool(want[:at + later].isfinite().all())
    assert bool(out[:at + later].isfinite().all())
    assert float(((out - want)[:at + later].abs() / want[:at + later].abs()).max()) <= (d + 41) * 2.0 ** -23


def test_a_numerator_beyond_a_float_stays_an_infinity():
    """Two opposite keys with opposite values: the normaliser nearly cancels, the products don't, and overflow where the divisor is
    small.  All factors are powers of two, so that a value is its first part."""
    H, d, dv, T = 1, 64, 128, 150
    proj = torch.zeros(T, 2 * H * d + H * dv)
    proj[3, d], proj[3, 2 * d:] = 1.0, 2.0 ** 17
    proj[4, d], proj[4, 2 * d:] = -1.0, -2.0 ** 17
    proj[4, 2 * d + dv // 2:] = 2.0 ** 17                # (these columns cancel)
    proj[10, 0] = 2.0 ** 117
    gates = torch.cat([torch.zeros(T, H), torch.full((T, H), 40.0)], dim=1)
    (out, _), (want, _) = both(proj, H, d, dv, gates)
    assert bool(want[10, 0, :dv // 2].isinf().all()) and bool(want[:10].isfinite().all())
    assert torch.equal(out.isinf(), want.isinf()) and not bool(out.isnan().any())
    assert torch.equal(out.sign(), want.sign())


@pytest.mark.parametrize("what", ["start state", "keys"])
def test_the_normaliser_adds_up_without_loss(what):
    """n . q from terms of about 1,000 that cancel to between 2 and 4, behind numerators that don't: products with the start state's n (a first
    chunk from a state in the slot, no keys), and weighted products with keys (gates that weigh every key with one).  What is left is
    one rounding of a float or two each in the sum, its quotient and the numerator: 2^-20, where float sums would be off by 2^-12."""
    from tensorline_b200 import ops
    H, d, dv, T = 1, 128, 64, 200
    g = torch.Generator().manual_seed(5)
    proj = torch.zeros(T, 2 * d + dv)
    gates = torch.cat([torch.zeros(T, H), torch.full((T, H), 2000.0)], dim=1)      # no decay at all below a cap of 400
    state = torch.zeros(1, H * -(-dv // ops.scan_columns()) * ops.scan_state_floats(d, True))
    terms = (torch.randn(T, d - 1, generator=g) * 1000.0).float()
    if what == "keys":                                   # token t from 100 on sees the keys 0 .. 99, whose products are c
        c = (torch.randn(100, generator=g) * 1000.0).float()
        c[99] = 3.0 - c[:99].double().sum()
        proj[:100, d], proj[:, 0] = c, 1.0
        proj[:100, 2 * d:] = c.sign()[:, None]
        at, want = slice(100, 128), c.double().abs().sum() / (c.double().sum().abs() + 1e-6)
    else:
        S, n = torch.zeros(H, d, dv), torch.randn(H, d, generator=g)
        S[0, 0], n[0, 0], n[0, d - 1] = 1.0, 0.0, 1.0
        state = chunks.slot_rows(S, n, torch.zeros(H))[None].float()
        proj[:, 0], proj[:, 1:d] = 1.0, terms
        proj[:, d - 1] = 3.0 - (proj[:, :d - 1].double() @ n[0, :d - 1].double())
        at, want = slice(0, 128), 1.0 / ((proj[:128, :d].double() @ n[0].double()).abs() + 1e-6)[:, None]
    i32 = dict(dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(h_q_start=[0, T], scratch={}, pos=torch.arange(T, **i32), q_start=torch.tensor([0, T], **i32), slots=torch.zeros(1, **i32))
    out = torch.empty(T, H * dv, device="cuda")
    ops.linear_chunks(proj.cuda(), 0, d, 2 * d, H, d, dv, state.cuda(), ctx, out, gates=gates.cuda(), cap=400.0, den_eps=1e-6)
    assert float(((out[at].double().cpu() - want).abs() / want).max()) <= 2.0 ** -20


def test_a_weight_is_one_exponential(monkeypatch):
    """One key in the first 32 tokens of a head, seen from the next 32: an output is its weight, and the same float as in chunks of 64 (whose
    argument is rounded from doubles; here from pairs of floats, which may round the other way at a tie)."""
    from tensorline_b200 import ops
    H, d, dv, T = 16, 64, 64, 64
    proj = torch.zeros(T, 2 * H * d + H * dv)
    proj[:, :H * d:d] = 1.0
    for h in range(H):
        proj[2 * h, H * d + h * d] = 1.0
        proj[2 * h, 2 * H * d + h * dv:2 * H * d + (h + 1) * dv] = 1.0
    decay = 1.0 - 0.3 * torch.rand(H, generator=torch.Generator().manual_seed(1))
    wide = both(proj, H, d, dv, None, decay)[0][0]
    monkeypatch.setattr(ops, "WIDE_CHUNKS_BLOCKS", {False: 1 << 40, True: 1 << 40})
    narrow = both(proj, H, d, dv, None, decay)[0][0]
    assert float((wide[32:, :, 0] == narrow[32:, :, 0]).float().mean()) >= 0.99


@pytest.mark.parametrize("gated,H,d,dv,T", [(True, 8, 128, 256, 256), (True, 8, 64, 128, 300), (False, 8, 128, 256, 300), (False, 16, 64, 64, 512)])
def test_errors_are_no_larger_than_in_chunks_of_64(gated, H, d, dv, T, monkeypatch):
    """Sizes and distributions as the decoders have them, from a state of zero, against 64 bits: outputs (a token's and a head's error, the
    median of all) and states.  1.02: what is left of draws of this size."""
    from tensorline_b200 import ops
    g = torch.Generator().manual_seed(T)
    proj = torch.randn(T, 2 * H * d + H * dv, generator=g) * 0.9
    gates = torch.cat([torch.randn(T, H, generator=g) * 1.3 - 2, torch.randn(T, H, generator=g) * 1.3 + 3], dim=1) if gated else None
    decay = None if gated else torch.tensor([1.0 - 2.0 ** (-5 - 5 * i / (H - 1)) for i in range(H)])
    zero = torch.zeros(H, d, dv, dtype=torch.float64)
    o, S, n, m, _ = chunks.recurrence(proj.double(), gates.double() if gated else None, decay, H, d, dv, zero, zero[:, :, 0] if gated else None,
                                      zero[:, 0, 0] if gated else None, torch.arange(T), None, 0, False, 15.0, d ** -0.5, 1.0, 1e-6)
    o, S = o.view(T, H, dv), chunks.slot_rows(S, n, m)
    errors = []
    for least in (0, 1 << 40):
        monkeypatch.setattr(ops, "WIDE_CHUNKS_BLOCKS", {False: least, True: least})
        out, state = both(proj, H, d, dv, gates, decay, d ** -0.5)[0]
        errors.append((float(((out.double().cpu() - o).norm(dim=-1) / o.norm(dim=-1)).median()), float((state[0].double().cpu() - S).norm() / S.norm())))
    for err, base in zip(*errors):
        assert err <= 1.02 * base, errors
