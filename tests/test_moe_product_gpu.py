"""The experts' products of long steps at the edges of their tiles: empty runs, runs around a tile's width, matrices that end inside a
tile, every epilogue; against float64 sums of the same bfloat16 values.  Bounds: a result is rounded once to bfloat16 (at most 2^-8 of
it), behind a gate both factors are rounded first (2^-8 each, of sums that may be off as below); a float sum of K products is off by less than K 2^-23 times the sum of the absolute products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tensorline_b200 import ops
    return ops


RUNS = [[5], [0, 1, 0, 17, 31, 33, 0], [256, 257, 3, 0, 512, 513, 64], [1] * 40, [300, 0, 40], [2, 0, 1031, 255]]


@pytest.mark.parametrize("runs", RUNS)
@pytest.mark.parametrize("K,F", [(64, 64), (200, 80), (1032, 336)])
@pytest.mark.parametrize("kind", ["plain", "relu_squared", "silu", "gelu_tanh", "swish_clamped"])
def test_runs_of_rows_times_their_own_matrices(ops, runs, K, F, kind):
    g = torch.Generator().manual_seed(len(runs) * K + F)
    E, P = len(runs), sum(runs) + 3                      # rows behind the last run (identity entries) are left alone
    gated = kind not in ("plain", "relu_squared")
    R = 2 * F if gated else F
    x = torch.randn(P, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, R, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    offsets = torch.tensor([0] + torch.tensor(runs).cumsum(0).tolist() + [P], dtype=torch.int32).cuda()
    out = torch.full((P, F), 7.0, dtype=torch.bfloat16, device="cuda")
    act = ("swish_clamped", 1.5, 1.7) if kind == "swish_clamped" else None if kind == "plain" else kind
    ops.moe_product(x, w, offsets, out, act=act, gated=gated)
    ops.check_device_status()
    assert bool((out[P - 3:] == 7.0).all())
    at = 0
    for e, n in enumerate(runs):
        if n == 0:
            continue
        xe, we = x[at:at + n].double(), w[e].double()
        z, size = xe @ we.T, xe.abs() @ we.abs().T * K * 2.0 ** -23
        got = out[at:at + n].double()
        if kind == "plain":
            assert bool(((got - z).abs() <= z.abs() * 2.0 ** -8 + 2 * size).all())
        elif kind == "relu_squared":
            want = z.clamp_min(0) ** 2
            assert bool(((got - want).abs() <= want * 4 * 2.0 ** -8 + 4 * z.abs() * size + size).all())
        else:
            a, b = z[:, :F], z[:, F:]
            da, db = a.abs() * 2.0 ** -8 + 2 * size[:, :F], b.abs() * 2.0 ** -8 + 2 * size[:, F:]
            if kind == "swish_clamped":
                ga = a.clamp_max(1.5)
                f, u = ga * torch.sigmoid(1.7 * ga), b.clamp(-1.5, 1.5) + 1.0
            else:
                f, u = a * torch.sigmoid(a) if kind == "silu" else torch.nn.functional.gelu(a, approximate="tanh"), b
            want = f * u                                 # the gates' slopes are below 1.2
            assert bool(((got - want).abs() <= 1.2 * da * u.abs() + f.abs() * db + 1.2 * da * db + want.abs() * 2.0 ** -8 + 1e-6).all())
        at += n


def test_columns_that_are_no_multiple_of_anything(ops):
    g = torch.Generator().manual_seed(2)
    x, w = torch.randn(70, 72, generator=g).to(torch.bfloat16).cuda(), torch.randn(2, 133, 72, generator=g).to(torch.bfloat16).cuda()
    out = torch.empty(70, 133, dtype=torch.bfloat16, device="cuda")
    ops.moe_product(x, w, torch.tensor([0, 37, 70], dtype=torch.int32).cuda(), out)
    want = torch.cat([x[:37].double() @ w[0].double().T, x[37:].double() @ w[1].double().T])
    assert bool(((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-3).all())
    assert not ops.core().tl_moe_product_takes(2, 72, 133, 1) and not ops.core().tl_moe_product_takes(2, 71, 133, 0)


@pytest.mark.parametrize("kind", ["plain", "relu_squared", "silu", "gelu_tanh", "swish_clamped"])
def test_sums_that_are_not_rounded_before_the_activation(ops, kind):
    g = torch.Generator().manual_seed(5)
    runs, K, F, gated = [1, 0, 40, 7], 520, 96, kind not in ("plain", "relu_squared")
    x = torch.randn(48, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(4, 2 * F if gated else F, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    out = torch.empty(48, F, dtype=torch.float32 if kind == "plain" else torch.bfloat16, device="cuda")
    offsets = torch.tensor([0] + torch.tensor(runs).cumsum(0).tolist(), dtype=torch.int32).cuda()
    ops.moe_product(x, w, offsets, out, act=("swish_clamped", 1.5, 1.7) if kind == "swish_clamped" else None if kind == "plain" else kind, gated=gated, raw=True)
    z = torch.cat([x[a:b].double() @ w[e].double().T for e, (a, b) in enumerate(zip(offsets.tolist(), offsets.tolist()[1:]))])
    a, b = z[:, :F], z[:, -F:]
    ga = a.clamp_max(1.5)
    want = {"plain": lambda: z, "relu_squared": lambda: z.clamp_min(0) ** 2, "silu": lambda: a * torch.sigmoid(a) * b,
            "gelu_tanh": lambda: torch.nn.functional.gelu(a, approximate="tanh") * b,
            "swish_clamped": lambda: ga * torch.sigmoid(1.7 * ga) * (b.clamp(-1.5, 1.5) + 1.0)}[kind]()
    assert bool(((out.double() - want).abs() <= want.abs() * (0 if kind == "plain" else 1.001 * 2.0 ** -8) + K * 2.0 ** -23 * 8).all())


@pytest.mark.parametrize("few", [False, True])
@pytest.mark.parametrize("gated,shared,on_input", [(True, True, False), (False, False, False), (True, False, True)])
def test_long_steps_agree_with_streamed_experts(ops, gated, shared, on_input, few, monkeypatch):
    """A step through the sorted runs and the same step token by token: roundings to bfloat16 in between are all that differs."""
    from tensorline_b200.parts import FEED_FORWARDS, PartSpec, Runtime
    from tensorline_b200.parts import moe
    from types import SimpleNamespace
    part = FEED_FORWARDS.build(PartSpec("routed_experts", dict(hidden=256, inner=192, experts=6, top=3, gated=gated, router_bias=False,
                                                               activation="silu" if gated else "relu_squared", shared_inner=192 if shared else None,
                                                               weight_on="input" if on_input else "output")), Runtime(torch.device("cuda", 0), torch.bfloat16, 16))
    g = torch.Generator().manual_seed(1)
    part.bind({n: (torch.randn(s.shape, generator=g) * 0.08).to(torch.bfloat16).cuda() for n, s in part.expected_tensors("l").items()}, "l")
    h = torch.randn(77, 256, generator=g).to(torch.bfloat16).cuda()
    ctx = SimpleNamespace(graph_max_ctx=0)
    if few:                                              # (weights on the input: streamed both times) the step could be streamed and is sorted all the same
        monkeypatch.setattr(moe, "STREAM_MAX_TOKENS", 100)
        monkeypatch.setattr(moe, "SORT_MIN_BYTES", -1e9)
    long = part.forward(h, ctx)
    monkeypatch.setattr(moe, "STREAM_MAX_TOKENS", 100)
    monkeypatch.setattr(moe, "SORT_MIN_BYTES", 1e12)
    short = part.forward(h, ctx)
    ops.check_device_status()
    assert float((long.float() - short.float()).norm() / short.float().norm()) <= (2.0 ** -9 if few else 2.0 ** -7)      # few: only roundings that fall on the other side; else three more of 2^-8 at most


def routed(hidden, inner, experts, top, **more):
    from tensorline_b200.parts import FEED_FORWARDS, PartSpec, Runtime
    part = FEED_FORWARDS.build(PartSpec("routed_experts", dict(hidden=hidden, inner=inner, experts=experts, top=top, router_bias=False, **more)),
                               Runtime(torch.device("cuda", 0), torch.bfloat16, 16))
    g = torch.Generator().manual_seed(1)
    part.bind({n: (torch.randn(s.shape, generator=g) * 0.08).to(torch.bfloat16).cuda() for n, s in part.expected_tensors("l").items()}, "l")
    return part


def captured(part, h):
    from types import SimpleNamespace
    ctx = SimpleNamespace(graph_max_ctx=4096)
    part.forward(h, ctx)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = part.forward(h, ctx)
    graph.replay()
    torch.cuda.synchronize()
    return y


@pytest.mark.parametrize("tokens", [8, 40, 64])
@pytest.mark.parametrize("more", [dict(experts=512, top=8), dict(experts=373, top=16), dict(experts=300, identity=212, top=8, scoring="softmax_share"),
                                  dict(experts=256, identity=16, top=8, scoring="softmax_share"), dict(experts=8, top=2)])
def test_captured_steps_take_every_router(ops, more, tokens, monkeypatch):
    """Decode steps are captured at any number of tokens, whatever the router: more entries than the sort takes, identities among them.
    Streamed and, as far as the sort goes, through sorted runs: nothing is rounded in one that is not in the other, but the other way now and then."""
    from tensorline_b200.parts import moe
    part = routed(256, 64, gated=True, activation="silu", **more)
    h = torch.randn(tokens, 256, generator=torch.Generator().manual_seed(tokens)).to(torch.bfloat16).cuda()
    monkeypatch.setattr(moe, "SORT_MIN_BYTES", -1e12)
    monkeypatch.setattr(moe, "SORT_MIN_BYTES_LONG", -1e12)
    y = captured(part, h)
    monkeypatch.setattr(moe, "SORT_MIN_BYTES", 1e12)
    monkeypatch.setattr(moe, "SORT_MIN_BYTES_LONG", 1e12)
    streamed = captured(part, h)
    ops.check_device_status()
    assert float((y.float() - streamed.float()).norm() / streamed.float().norm()) <= 2.0 ** -9


def test_gates_that_the_sorted_products_do_not_have(ops, monkeypatch):
    """relu(gate)^2 * up: steps of few tokens and captured ones are streamed, whatever sorting would save; longer ones are refused."""
    from types import SimpleNamespace
    from tensorline_b200.parts import moe
    part = routed(256, 64, experts=8, top=2, gated=True, activation="relu_squared")
    h = torch.randn(77, 256, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).cuda()
    monkeypatch.setattr(moe, "SORT_MIN_BYTES", -1e12)
    monkeypatch.setattr(moe, "SORT_MIN_BYTES_LONG", -1e12)
    z = h.float() @ part.w_router.float().T
    wts, idx = z.topk(2, dim=1)
    wts = wts.softmax(dim=1)
    want = torch.zeros(77, 256, device="cuda")
    for t in range(77):
        for j in range(2):
            gate, up = (part.w_up[idx[t, j]].float() @ h[t].float()).split(64)
            want[t] += wts[t, j] * (part.w_down[idx[t, j]].float() @ (gate.clamp_min(0) ** 2 * up))
    for y in (captured(part, h), torch.cat([part.forward(x, SimpleNamespace(graph_max_ctx=0)) for x in h.split(32)])):
        assert float((y.float() - want).norm() / want.norm()) <= 2.0 ** -7      # two roundings to bfloat16, each 2^-9 or less, and few sums' order
    with pytest.raises(ops.KernelError):
        part.forward(h, SimpleNamespace(graph_max_ctx=0))


@pytest.mark.parametrize("act", ["silu", "swish_clamped"])
def test_far_gates_of_few_tokens_are_divided_exactly(ops, act):
    """x / (1 + e^-x) where the divisor is above 2^126: small but no zero, and an up value brings it back into sight.  Against the
    formula in float64; three roundings of bfloat16 values and floats (2^-8 and less) beside the exponential's argument."""
    x = torch.zeros(5, 64)
    x[:, 0], x[:, 1] = torch.tensor([-80.0, -87.0, -87.5, -88.0, -88.5]), 2.0 ** 100
    w = torch.zeros(1, 32, 64)
    w[0, :16, 0], w[0, 16:, 1] = 1.0, 1.0
    x, w = x.to(torch.bfloat16).cuda(), w.to(torch.bfloat16).cuda()
    out = torch.empty(5, 16, dtype=torch.bfloat16, device="cuda")
    clamped = act == "swish_clamped"
    ops.moe_product(x, w, torch.tensor([0, 5], dtype=torch.int32).cuda(), out, act=("swish_clamped", 1e38, 1.0) if clamped else act, gated=True, raw=True)
    z = x[:, 0].double()
    want = (z / (1.0 + torch.exp(-z)) * (2.0 ** 100 + (1.0 if clamped else 0.0)))[:, None]
    assert float(((out.double() - want).abs() / want.abs()).max()) <= 2.0 ** -7


@pytest.mark.parametrize("tokens,inner,sorts", [(40, 64, False), (64, 64, False), (64, 1024, True)])
def test_captured_steps_over_small_experts_are_streamed(ops, tokens, inner, sorts, monkeypatch):
    """Above STREAM_MAX_TOKENS too a captured step is sorted only where that is the faster way."""
    part = routed(256, inner, experts=8, top=2, gated=True, activation="silu")
    h = torch.randn(tokens, 256, generator=torch.Generator().manual_seed(tokens)).to(torch.bfloat16).cuda()
    calls, sort = [], ops.moe_sort
    monkeypatch.setattr(ops, "moe_sort", lambda *a: calls.append(a) or sort(*a))
    captured(part, h)
    assert bool(calls) == sorts
