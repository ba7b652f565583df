"""What this engine spends its time on: the steps, layers and mixers that its performance is measured by.

`listed()` are fixed cases, `draw(rng)` gives more of the same ranges.  Sizes are those of the benchmark: the published Qwen2.5
layer sizes for the dense decoder, and the "2k" sizes at which `bench.py --design` runs the other decoders' parts.

    decode_step      a whole decode step of a short Qwen2 model through the runner's decode graph, logits of every request
    dense_block      one layer (attention and feed-forward) of the dense decoder over the paged cache: prompt portions on cached
                     tokens, single decoded tokens, or both, in bfloat16 or in the true 32-bit engine
    memory           one mixer that carries a state: mlstm, retention, hgrn2, gated_delta; prompt portions, or single tokens
                     from a CUDA graph (as the engine decodes)
    experts          one routed feed-forward: a prompt step, or single tokens from a CUDA graph

Single bfloat16 tokens run from a captured graph because that is how the engine runs them.  Nothing here is tuned to a case:
weights are random at the scale of the random-weights mode, norm outputs are unit normal, gates and decays are spread as the
papers initialise them, so that states remember from a few to many hundreds of tokens.
"""
from __future__ import annotations

import zlib

import torch

from tensorline_b200 import Engine, Qwen2Config
from tensorline_b200.engine.runner import StepContext, StepEntry
from tensorline_b200.parts import BLOCKS, FEED_FORWARDS, MIXERS, KVCacheView, PartSpec, Runtime, StateView
from tensorline_b200.parts.linear import resolve

PAGE = 16
SEVEN_B = dict(hidden=3584, heads=28, kv_heads=4, inter=18944)
FOURTEEN_B = dict(hidden=5120, heads=40, kv_heads=8, inter=13824)
MEMORY = dict(hidden=2048, heads=8, dim=128, vdim=256)
EXPERTS = dict(hidden=2048, inner=1024, experts=32, top=4)


def listed():
    return [
        # the headline: eight requests decode one token each near the end of a 4,096-token context
        dict(name="decode_step_8", kind="decode_step", layers=4, vocab=152064, batch=8, context=4090, **SEVEN_B),
        # a whole 2,048-token prompt through one layer
        dict(name="dense_prompt_2048", kind="dense_block", dtype="bfloat16", portion=2048, cached=0, singles=0, context=0, **SEVEN_B),
        # continuous batching: a prompt's second portion beside 48 requests that decode
        dict(name="dense_mixed_512", kind="dense_block", dtype="bfloat16", portion=464, cached=1024, singles=48, context=1500, **FOURTEEN_B),
        # the true 32-bit engine as logit checks and replays use it: a portion on cached tokens beside three decoding requests ...
        dict(name="float32_portion_333", kind="dense_block", dtype="float32", portion=333, cached=700, singles=3, context=900, **SEVEN_B),
        # ... and a replay token by token
        dict(name="float32_tokens_4", kind="dense_block", dtype="float32", portion=0, cached=0, singles=4, context=1800, **SEVEN_B),
        # the matrix memory: a whole prompt, and one request that decodes (the smallest call)
        dict(name="mlstm_prompt_2048", kind="memory", mixer="mlstm", tokens=2048, requests=1, graph=False, **MEMORY),
        dict(name="mlstm_token_1", kind="memory", mixer="mlstm", tokens=1, requests=1, graph=True, **MEMORY),
        # retention: three prompts of unequal length in one step
        dict(name="retention_prompts_1650", kind="memory", mixer="retention", tokens=1650, requests=3, graph=False, **MEMORY),
        # the gated delta rule behind its short convolutions: a whole prompt
        dict(name="delta_prompt_2048", kind="memory", mixer="gated_delta", tokens=2048, requests=1, graph=False, **MEMORY),
        # HGRN2: two prompts in one step
        dict(name="hgrn2_prompts_1911", kind="memory", mixer="hgrn2", tokens=1911, requests=2, graph=False, **MEMORY),
        # routed experts beside a shared one: a prompt step, and eight requests that decode
        dict(name="experts_prompt_2048", kind="experts", tokens=2048, gated=True, shared=True, graph=False, **EXPERTS),
        dict(name="experts_tokens_8", kind="experts", tokens=8, gated=True, shared=True, graph=True, **EXPERTS),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["decode_step", "dense_block", "dense_block", "memory", "memory", "memory", "experts", "experts"])
    if kind == "decode_step":
        return dict(kind=kind, layers=rng.randint(1, 3), vocab=rng.choice([32000, 152064]), batch=_log_int(rng, 1, 64),
                    context=_log_int(rng, 64, 4000), **SEVEN_B)
    if kind == "dense_block":
        if rng.random() < 0.4:
            width = rng.choice([dict(hidden=2048, heads=16, kv_heads=4, inter=5504), SEVEN_B])
            portion = rng.choice([0, _log_int(rng, 2, 330)])
            return dict(kind=kind, dtype="float32", portion=portion, cached=rng.randint(0, 700) if portion else 0,
                        singles=rng.randint(0, 3) if portion else rng.randint(1, 16), context=_log_int(rng, 30, 1800), **width)
        width = rng.choice([dict(hidden=2048, heads=16, kv_heads=4, inter=5504), SEVEN_B, FOURTEEN_B])
        singles = rng.choice([0, _log_int(rng, 1, 64)])
        return dict(kind=kind, dtype="bfloat16", portion=_log_int(rng, 40, 2048), cached=rng.choice([0, rng.randint(1, 2048)]),
                    singles=singles, context=_log_int(rng, 60, 2000) if singles else 0, **width)
    if kind == "memory":
        graph = rng.random() < 0.25
        requests = _log_int(rng, 1, 64) if graph else rng.randint(1, 4)
        heads = rng.choice([4, 8, 16])
        return dict(kind=kind, mixer=rng.choice(["mlstm", "retention", "gated_delta", "gated_delta", "hgrn2"]),
                    tokens=requests if graph else _log_int(rng, 40 * requests, 2048), requests=requests, graph=graph,
                    hidden=rng.choice([1024, 1536, 2048]), heads=heads, dim=rng.choice([64, 96, 128] if heads > 4 else [128, 256]),
                    vdim=rng.choice([64, 128, 256] if heads < 16 else [64, 128]))
    graph = rng.random() < 0.35
    return dict(kind=kind, tokens=_log_int(rng, 1, 32) if graph else _log_int(rng, 40, 2048), gated=rng.random() < 0.6,
                shared=rng.random() < 0.5, graph=graph, hidden=rng.choice([1024, 1536, 2048]), inner=64 * rng.randint(8, 16),
                experts=rng.choice([8, 16, 24, 32]), top=rng.randint(2, 4))


# ------------------------------------------------------------------------------------------ inputs
def _rand(seed, name, shape, scale=1.0, mean=0.0, dtype=torch.bfloat16, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed((int(seed) << 20) ^ zlib.crc32(name.encode()))
    return (torch.empty(shape, dtype=torch.float32, device=device).normal_(mean, scale, generator=g)).to(dtype)


def _weights(part, seed, prefix):
    """Random weights as the engine's random-weights mode draws them, and gates, decays and taps as the papers start them."""
    out = {}
    for name, spec in part.expected_tensors(prefix).items():
        leaf = name[len(prefix) + 1:]
        scale, mean, dtype = 0.02, 0.0, torch.bfloat16
        if spec.init == "ones":
            scale, mean = 0.1, 1.0
        if leaf.endswith(".conv"):
            scale = 0.5
        elif leaf == "A_log":
            scale, mean, dtype = 1.2, -2.0, torch.float32
        elif leaf == "dt_bias":
            scale, mean, dtype = 1.0, -1.0, torch.float32
        elif leaf == "f.b":
            scale, mean = 1.0, 3.0
        elif leaf == "i.b":
            scale, mean = 1.0, -2.0
        out[name] = _rand(seed, name, spec.shape, scale, mean, dtype)
        if leaf == "lower":
            out[name] = (out[name].float().mul(40.0).sigmoid() * 0.9).to(torch.bfloat16)
    return out


def _lengths(total, requests):
    """`total` tokens over `requests` of unequal length, each at least one."""
    w = [2.0 ** -i for i in range(requests)]
    out = [max(1, int(total * x / sum(w))) for x in w]
    out[0] += total - sum(out)
    return out


def _context(lengths, starts, tables, decode, graph_ctx=0):
    """The description of a step with `lengths[i]` tokens of request i, which stands at position `starts[i]`."""
    B, T = len(lengths), sum(lengths)
    q_start = [0]
    for n in lengths:
        q_start.append(q_start[-1] + n)
    pos = [s + i for n, s in zip(lengths, starts) for i in range(n)]
    slot = [b for b, n in enumerate(lengths) for _ in range(n)]

    def dev(a):
        return torch.tensor(a, dtype=torch.int32, device="cuda")
    return StepContext(T=T, B=B, ids=dev([0] * T), pos=dev(pos), req_slot=dev(slot), q_start=dev(q_start), start_pos=dev(starts),
                       slots=dev(list(range(B))), want_rows=dev([]), tables=tables, page_size=PAGE, decode_only=decode,
                       max_q_len=max(lengths), max_ctx=max(s + n for s, n in zip(starts, lengths)), h_q_start=q_start,
                       h_start_pos=list(starts), h_slots=list(range(B)), graph_max_ctx=graph_ctx)


def _captured(call):
    """`call` as a CUDA graph, the way the runner captures a decode step; returns (graph, its outputs)."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            call()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = call()
    return graph, out


def _dense_requests(case):
    """(tokens, tokens already cached) of every request of a dense step: the decoding ones first, then the portion's."""
    n, ctx = case["singles"], case["context"]
    reqs = [(1, max(1, ctx - 37 * (i % 7))) for i in range(n)]
    return reqs + ([(case["portion"], case["cached"])] if case["portion"] else [])


def _pages(reqs, seed):
    """A block table with every request's pages in random places of one pool; (table, pages of the pool)."""
    need = [-(-(n + c) // PAGE) for n, c in reqs]
    total = sum(need)
    perm = torch.randperm(total, generator=torch.Generator().manual_seed(seed)).to(torch.int32)
    table = torch.full((len(reqs) + 1, max(need)), total, dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n]
        at += n
    return table.cuda(), total


def _dense_spec(case):
    norm = PartSpec("rms_norm", {"dim": case["hidden"], "eps": 1e-6})
    mixer = PartSpec("paged_attention", {"hidden": case["hidden"], "num_heads": case["heads"], "num_kv_heads": case["kv_heads"],
                                         "head_dim": 128, "qkv_bias": True, "position": PartSpec("rotary_half", {"theta": 1e6})})
    ff = PartSpec("gated_mlp", {"hidden": case["hidden"], "intermediate": case["inter"], "activation": "silu"})
    return PartSpec("pre_norm", {"mixer": mixer, "feed_forward": ff, "norm1": norm, "norm2": norm})


def _memory_spec(case):
    p = {"hidden": case["hidden"], "num_heads": case["heads"], "head_dim": case["dim"], "v_head_dim": case["vdim"], "norm_eps": 1e-5}
    if case["mixer"] == "mlstm":
        p["gate_cap"] = 15.0
    elif case["mixer"] == "retention":
        H = case["heads"]
        p["decay"] = [1.0 - 2.0 ** (-5 - 5 * i / max(1, H - 1)) for i in range(H)]
        p["position"] = PartSpec("rotary_half", {"theta": 1e6, "rotary_dim": case["dim"]})
    elif case["mixer"] == "gated_delta":
        p["num_qk_heads"] = case["heads"] // 2
        p["taps"] = 4
    return PartSpec(case["mixer"], p)


def _experts_spec(case):
    return PartSpec("routed_experts", {
        "hidden": case["hidden"], "inner": case["inner"], "experts": case["experts"], "top": case["top"], "gated": case["gated"],
        "activation": "silu" if case["gated"] else "relu_squared", "router_bias": False, "scoring": "softmax_chosen",
        "shared_inner": case["inner"] if case["shared"] and case["gated"] else None})


def _qwen2(case):
    return Qwen2Config.from_dict(dict(
        architectures=["Qwen2ForCausalLM"], num_hidden_layers=case["layers"], hidden_size=case["hidden"],
        num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=128, intermediate_size=case["inter"],
        vocab_size=case["vocab"], rope_theta=1e6, rms_norm_eps=1e-6, tie_word_embeddings=False, use_sliding_window=False,
        max_position_embeddings=32768, hidden_act="silu", eos_token_id=1))


def _qwen2_weights(cfg, seed):
    from tensorline_b200.models import expected_tensors
    return {name: _rand(seed, name, spec.shape, *((0.1, 1.0) if spec.init == "ones" else (0.02, 0.0)))
            for name, spec in expected_tensors(cfg).items() if not spec.optional}


def _decode_tokens(case, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, case["vocab"], (case["batch"],), generator=g).tolist()


def _decode_kv(case, seed, layer):
    """Keys and values of the tokens before the step: [pages, kv heads, PAGE, 128] each; request i holds its own run of pages."""
    pages = case["batch"] * -(-(case["context"] + 1) // PAGE)
    shape = (pages, case["kv_heads"], PAGE, 128)
    return _rand(seed, f"k{layer}", shape), _rand(seed, f"v{layer}", shape)


# ------------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    return {"decode_step": _prepare_decode, "dense_block": _prepare_dense, "memory": _prepare_memory,
            "experts": _prepare_experts}[case["kind"]](case, seed)


def _prepare_decode(case, seed):
    cfg = _qwen2(case)
    batch, ctx = case["batch"], case["context"]
    per = -(-(ctx + 1) // PAGE)
    eng = Engine(cfg, dtype="bfloat16", weights=_qwen2_weights(cfg, seed), block_size=PAGE, num_blocks=batch * per,
                 max_num_seqs=batch, max_model_len=per * PAGE, prefix_caching=False)
    reqs = list(range(batch))
    for i in reqs:
        assert eng.cache.admit(i) is not None
        eng.runner.start_request(i, ctx)                    # its first `ctx` tokens are in its pages
        assert eng.cache.grow(i, 0, ctx + 1)
    order = [p for i in reqs for p in eng.cache.pages(i)]   # the pool's pages in the order of `_decode_kv`
    order = torch.tensor(order, device="cuda")
    for layer in range(case["layers"]):
        view = eng.runner.caches[layer]
        k, v = _decode_kv(case, seed, layer)
        view.k[order], view.v[order] = k, v
    entries = [StepEntry(i, [t], [0]) for i, t in enumerate(_decode_tokens(case, seed))]
    eng.runner.step_graph(entries)                          # the step's graph is captured once and kept
    return {"case": case, "engine": eng, "entries": entries}


def _prepare_dense(case, seed):
    act = getattr(torch, case["dtype"])
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), act, PAGE)
    block = BLOCKS.build(_dense_spec(case), rt)
    block.bind(_weights(block, seed, "l"), "l")
    reqs = _dense_requests(case)
    table, total = _pages(reqs, seed)
    k, v = _dense_kv(case, seed, total)
    ctx = _context([n for n, _ in reqs], [c for _, c in reqs], [table], all(n == 1 for n, _ in reqs))
    T = ctx.T
    return {"case": case, "part": block, "ctx": ctx, "cache": KVCacheView(k.to(act), v.to(act), 0),
            "x": _rand(seed, "x", (T, case["hidden"]), dtype=torch.float32), "pending": _rand(seed, "pending", (T, case["hidden"]), dtype=act)}


def _dense_kv(case, seed, total):
    shape = (total + 1, case["kv_heads"], PAGE, 128)
    return _rand(seed, "k", shape), _rand(seed, "v", shape)


PROMPT_BEFORE_GRAPH = 48


def _prepare_memory(case, seed):
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), torch.bfloat16, PAGE)
    part = MIXERS.build(_memory_spec(case), rt)
    part.bind(_weights(part, seed, "l"), "l")
    n = case["requests"]
    lengths = _lengths(case["tokens"], n)
    dtypes = {"float32": torch.float32}

    def view(need):
        return StateView(torch.zeros((n + 1,) + tuple(need.shape), dtype=dtypes[need.dtype], device="cuda"))
    need = part.cache_need()
    cache = {k: view(v) for k, v in need.items()} if isinstance(need, dict) else view(need)
    state = {"case": case, "part": part, "cache": cache}
    h = _rand(seed, "h", (case["tokens"], case["hidden"]))
    if not case["graph"]:
        state.update(h=h, ctx=_context(lengths, [0] * n, [], False))
        return state
    ctx = _context([1] * n, [PROMPT_BEFORE_GRAPH] * n, [], True, graph_ctx=4096)
    state["graph"], state["out"] = _captured(lambda: part.forward(h, ctx, cache))
    state["keep"] = (h, ctx)
    for s in _states(cache):                                # what the captured calls left behind
        s.zero_()
    before = _rand(seed, "before", (PROMPT_BEFORE_GRAPH * n, case["hidden"]))
    part.forward(before, _context([PROMPT_BEFORE_GRAPH] * n, [0] * n, [], False), cache)
    return state


def _states(cache):
    return [v.state for _, v in sorted(cache.items())] if isinstance(cache, dict) else [cache.state]


def _prepare_experts(case, seed):
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), torch.bfloat16, PAGE)
    part = FEED_FORWARDS.build(_experts_spec(case), rt)
    part.bind(_weights(part, seed, "l"), "l")
    T = case["tokens"]
    h = _rand(seed, "h", (T, case["hidden"]))
    state = {"case": case, "part": part, "h": h}
    if case["graph"]:
        ctx = _context([1] * T, [100] * T, [], True, graph_ctx=4096)
        state["graph"], state["out"] = _captured(lambda: part.forward(h, ctx))
    else:
        ctx = _context([T], [0], [], False)
    state["ctx"] = ctx
    return state


# ------------------------------------------------------------------------------------------ run
@torch.inference_mode()
def run(state):
    case = state["case"]
    if case["kind"] == "decode_step":
        runner = state["engine"].runner
        for e in state["entries"]:
            runner.positions[e.rid] = case["context"]       # the same token again: the last step's place is overwritten
        return runner.step_graph(state["entries"])
    if case["kind"] == "dense_block":
        x = state["x"].clone()                              # the embedding's output; the block adds to it in place
        out = state["part"].forward(x, state["pending"], state["ctx"], state["cache"])
        return {"out": resolve(out), "stream": x}
    if case["kind"] == "memory":
        if case["graph"]:                                   # decoding: the state goes on from pass to pass
            state["graph"].replay()
            return {"out": state["out"], "state": [s[:-1] for s in _states(state["cache"])]}
        for s in _states(state["cache"]):                   # new requests: their slots start from zero
            s.zero_()
        out = state["part"].forward(state["h"], state["ctx"], state["cache"])
        return {"out": resolve(out), "state": [s[:-1] for s in _states(state["cache"])]}
    if case["graph"]:
        state["graph"].replay()
        return state["out"]
    return resolve(state["part"].forward(state["h"], state["ctx"]))


# ------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    if case["kind"] in ("decode_step", "dense_block"):
        H, d = case["hidden"], 128
        nq, nkv = case["heads"], case["kv_heads"]
        weights = (nq + 2 * nkv) * d * H + nq * d * H + 3 * H * case["inter"]
        if case["kind"] == "decode_step":
            b, ctx = case["batch"], case["context"]
            w = case["layers"] * weights + case["vocab"] * H
            kv = case["layers"] * b * (ctx + 1) * nkv * d * 2 * 2
            return {"bytes": 2 * w + kv + b * case["vocab"] * 4, "flops": 2 * b * w + case["layers"] * 4 * b * (ctx + 1) * nq * d}
        reqs = _dense_requests(case)
        T = sum(n for n, _ in reqs)
        item = 2 if case["dtype"] == "bfloat16" else 4
        pairs = sum(n * c + n * (n + 1) // 2 for n, c in reqs)
        kv = sum(n + c for n, c in reqs) * nkv * d * 2 * item
        return {"bytes": 2 * weights + kv + T * H * (4 + 4 + 2 * item), "flops": 2 * T * weights + 4 * pairs * nq * d}
    if case["kind"] == "memory":
        W, H, d, dv, T = case["hidden"], case["heads"], case["dim"], case["vdim"], case["tokens"]
        nqk = H // 2 if case["mixer"] == "gated_delta" else H
        rows = 2 * nqk * d + H * dv + (0 if case["mixer"] == "hgrn2" else H * dv)
        weights = rows * W + W * H * dv
        state = case["requests"] * H * d * dv * 4
        per_token = H * d * dv * (6 if case["mixer"] == "gated_delta" else 4)
        return {"bytes": 2 * weights + T * W * 4 + state * (2 if case["graph"] else 1), "flops": T * (2 * weights + per_token)}
    W, F, T, top = case["hidden"], case["inner"], case["tokens"], case["top"]
    expert = (3 if case["gated"] else 2) * W * F
    used = case["experts"] * (1 - (1 - top / case["experts"]) ** T)      # experts that some token chose, on average
    shared = expert if case["shared"] and case["gated"] else 0
    return {"bytes": 2 * (used * expert + shared) + T * W * 4, "flops": 2 * T * (top * expert + shared + case["experts"] * W)}


def tolerance(case):
    """Rounding to bfloat16 between the steps of a part, where there is any; else float32 sums in another order."""
    if case["kind"] == "dense_block" and case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["kind"] == "decode_step":
        return {"rel": 0.03}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------ the same in 64 bits
@torch.no_grad()
def exact(case, seed):
    return {"decode_step": _exact_decode, "dense_block": _exact_dense, "memory": _exact_memory,
            "experts": _exact_experts}[case["kind"]](case, seed)


def _norm64(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _rotate64(x, pos, theta, dim):
    """x [T, heads, dim]; pairs (i, i + dim / 2), angles from float32 frequencies as the engine defines them."""
    i = torch.arange(0, dim, 2, dtype=torch.float64)
    f = (float(theta) ** (-i / dim)).to(torch.float32).double().to(x.device)
    a = (pos.double()[:, None] * f)[:, None, :]
    c, s = torch.cos(a), torch.sin(a)
    x1, x2 = x[..., :dim // 2], x[..., dim // 2:]
    return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], dim=-1)


def _attend64(q, k, v, start, groups):
    """q [n, nq, d] at positions start.., k and v [m, nkv, d] of positions 0..m - 1."""
    n, nq, d = q.shape
    out = torch.empty_like(q)
    at = torch.arange(start, start + n, device=q.device)[:, None]
    mask = torch.arange(k.shape[0], device=q.device)[None, :] > at
    for h in range(nq):
        s = (q[:, h] @ k[:, h // groups].T) * d ** -0.5
        out[:, h] = torch.softmax(s.masked_fill_(mask, -float("inf")), dim=-1) @ v[:, h // groups]
    return out.reshape(n, nq * d)


def _layer64(case, get, x, reqs, old):
    """One dense layer in 64 bits: (addend, stream).  `get(name)`: a weight; `old(i)`: request i's earlier keys and values."""
    nq, nkv, d = case["heads"], case["kv_heads"], 128
    h = _norm64(x, get("input_layernorm.weight"), 1e-6)

    def lin(name, y):
        return y @ get(f"self_attn.{name}_proj.weight").double().T
    q, k, v = (lin(n, h) + get(f"self_attn.{n}_proj.bias").double() for n in "qkv")
    rows, at = [], 0
    for i, (n, c) in enumerate(reqs):
        sl = slice(at, at + n)
        pos = torch.arange(c, c + n, device=x.device)
        qi = _rotate64(q[sl].view(n, nq, d), pos, 1e6, d)
        ki = _rotate64(k[sl].view(n, nkv, d), pos, 1e6, d)
        ko, vo = old(i)
        rows.append(_attend64(qi, torch.cat([ko, ki]), torch.cat([vo, v[sl].view(n, nkv, d)]), c, nq // nkv))
        at += n
    x = x + lin("o", torch.cat(rows))
    h = _norm64(x, get("post_attention_layernorm.weight"), 1e-6)
    g, u = h @ get("mlp.gate_proj.weight").double().T, h @ get("mlp.up_proj.weight").double().T
    return (g * torch.sigmoid(g) * u) @ get("mlp.down_proj.weight").double().T, x


def _exact_dense(case, seed):
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), getattr(torch, case["dtype"]), PAGE)
    w = _weights(BLOCKS.build(_dense_spec(case), rt), seed, "l")
    reqs = _dense_requests(case)
    table, total = _pages(reqs, seed)
    k, v = _dense_kv(case, seed, total)

    def old(i):
        c = reqs[i][1]
        idx = table[i, :-(-c // PAGE)].long()
        return tuple(t[idx].permute(0, 2, 1, 3).reshape(idx.numel() * PAGE, case["kv_heads"], 128)[:c].double() for t in (k, v))
    T = sum(n for n, _ in reqs)
    x = _rand(seed, "x", (T, case["hidden"]), dtype=torch.float32).double()
    x = x + _rand(seed, "pending", (T, case["hidden"]), dtype=getattr(torch, case["dtype"])).double()
    out, stream = _layer64(case, lambda n: w["l." + n], x, reqs, old)
    return {"out": out, "stream": stream}


def _exact_decode(case, seed):
    w = _qwen2_weights(_qwen2(case), seed)
    b, ctx = case["batch"], case["context"]
    per = -(-(ctx + 1) // PAGE)
    x = w["model.embed_tokens.weight"][torch.tensor(_decode_tokens(case, seed), device="cuda")].double()
    for layer in range(case["layers"]):
        kv = _decode_kv(case, seed, layer)

        def old(i):
            return tuple(t[i * per:(i + 1) * per].permute(0, 2, 1, 3).reshape(-1, case["kv_heads"], 128)[:ctx].double() for t in kv)
        out, x = _layer64(case, lambda n: w[f"model.layers.{layer}.{n}"], x, [(1, ctx)] * b, old)
        x = x + out
    h = _norm64(x, w["model.norm.weight"], 1e-6)
    head = w["lm_head.weight"]
    return torch.cat([h @ part.double().T for part in head.split(16384)], dim=1)


def _state_rows(S, extra, m):
    """One request's matrices S [H, d, dv] (and, per head, a column `extra` [H, d] and a number m [H]) as a slot holds them: per head
    and slice of 16 columns, rows dealt out to threads, R consecutive rows each."""
    H, d, dv = S.shape
    R, IS = (4, 8) if d <= 32 else (8, 8) if d <= 64 else (8, 16) if d <= 128 else (8, 32)
    nz, cols = -(-dv // 16), 16 if extra is None else 17
    NT = -(-IS * cols // 32) * 32
    full = S.new_zeros(H, IS * R, nz * 16)
    full[:, :d, :dv] = S
    full = full.view(H, IS, R, nz, 16).permute(0, 3, 2, 4, 1)                   # [H, nz, R, column, IS]
    out = S.new_zeros(H, nz, R, NT)
    out[..., :16 * IS] = full.reshape(H, nz, R, 16 * IS)
    if extra is None:
        return out.reshape(-1)
    col = S.new_zeros(H, IS * R)
    col[:, :d] = extra
    out[..., 16 * IS:17 * IS] = col.view(H, 1, IS, R).permute(0, 1, 3, 2)
    tail = S.new_zeros(H, nz, 4)
    tail[..., 0] = m[:, None]
    return torch.cat([out.reshape(H, nz, -1), tail], dim=2).reshape(-1)


def _memory64(case, w, h, start=0, carry=None):
    """One request's tokens h [n, hidden] through the mixer: (y [n, hidden], carry)."""
    H, d, dv, kind = case["heads"], case["dim"], case["vdim"], case["mixer"]
    n = h.shape[0]
    get = {k[2:]: v.double() for k, v in w.items()}

    def proj(name, heads, size):
        return (h @ get[name].T).view(n, heads, size)
    S = carry["S"] if carry else h.new_zeros(H, d, dv)
    norm = carry["n"] if carry else h.new_zeros(H, d)
    m = carry["m"] if carry else h.new_zeros(H)
    kept = None
    o = h.new_empty(n, H, dv)
    pos = torch.arange(start, start + n, device=h.device)
    if kind == "gated_delta":
        nqk, taps = H // 2, 4
        raw = torch.cat([h @ get[k].T for k in "qkv"], dim=1)
        past = carry["kept"] if carry else raw.new_zeros(taps - 1, raw.shape[1])
        rows = torch.cat([past, raw])
        kept = rows[-(taps - 1):]
        cw = torch.cat([get[k + ".conv"] for k in "qkv"])
        c = sum(rows[j:j + n] * cw[:, j] for j in range(taps))
        c = c * torch.sigmoid(c)
        q, k, v = c[:, :nqk * d].view(n, nqk, d), c[:, nqk * d:2 * nqk * d].view(n, nqk, d), c[:, 2 * nqk * d:].view(n, H, dv)
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k = (x.repeat_interleave(H // nqk, dim=1) for x in (q * d ** -0.5, k))
        beta = torch.sigmoid(h @ get["b"].T)
        g = torch.exp(-torch.exp(get["A_log"]) * torch.nn.functional.softplus(h @ get["a"].T + get["dt_bias"]))
        for t in range(n):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hd,hde->he", k[t], S))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = torch.einsum("hd,hde->he", q[t], S)
        weight, gate, act = get["norm"].repeat(H), proj("g", H, dv), "silu"
    elif kind == "hgrn2":
        q, v = proj("q", H, d), proj("v", H, dv)
        q = q * torch.sigmoid(q)
        low = get["lower"].view(H, d)
        f = low + (1 - low) * torch.sigmoid(proj("f", H, d) + get["f.b"].view(H, d))
        for t in range(n):
            S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None, :]
            o[t] = torch.einsum("hd,hde->he", q[t], S)
        weight, gate, act = get["norm"].repeat(H), None, None
    else:
        q, k, v, gate = proj("q", H, d), proj("k", H, d), proj("v", H, dv), proj("g", H, dv)
        if kind == "retention":
            q, k = _rotate64(q, pos, 1e6, d), _rotate64(k, pos, 1e6, d) * d ** -0.5
            decay = torch.tensor([1.0 - 2.0 ** (-5 - 5 * i / max(1, H - 1)) for i in range(H)], dtype=torch.float32, device=h.device).double()
            for t in range(n):
                S = decay[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hd,hde->he", q[t], S)
            weight, act = None, "silu"
        else:
            q = q * d ** -0.5
            li = 15.0 * torch.tanh((h @ get["i"].T + get["i.b"]) / 15.0)
            lf = torch.nn.functional.logsigmoid(15.0 * torch.tanh((h @ get["f"].T + get["f.b"]) / 15.0))
            for t in range(n):
                new = torch.maximum(lf[t] + m, li[t])
                a, b = torch.exp(lf[t] + m - new), torch.exp(li[t] - new)
                m = new
                S = a[:, None, None] * S + b[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
                norm = a[:, None] * norm + b[:, None] * k[t]
                den = torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                o[t] = torch.einsum("hd,hde->he", q[t], S) / den[:, None]
            weight, act = get["norm"], "sigmoid"
    y = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5)).view(n, H * dv)
    if weight is not None:
        y = y * weight
    if gate is not None:
        gate = gate.reshape(n, H * dv)
        y = y * (torch.sigmoid(gate) * (gate if act == "silu" else 1.0))
    return y @ get["o"].T, {"S": S, "n": norm, "m": m, "kept": kept}


def _exact_memory(case, seed):
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), torch.bfloat16, PAGE)
    w = _weights(MIXERS.build(_memory_spec(case), rt), seed, "l")
    n = case["requests"]
    h = _rand(seed, "h", (case["tokens"], case["hidden"])).double()
    before = _rand(seed, "before", (PROMPT_BEFORE_GRAPH * n, case["hidden"])).double() if case["graph"] else None
    if case["graph"] and n > 16:
        return None                                         # too many short chains, one after the other
    ys, states, kept, at = [], [], [], 0
    for i, size in enumerate(_lengths(case["tokens"], n)):
        start, carry = 0, None
        if case["graph"]:
            start = PROMPT_BEFORE_GRAPH
            _, carry = _memory64(case, w, before[i * start:(i + 1) * start])
        y, carry = _memory64(case, w, h[at:at + size], start, carry)
        at += size
        ys.append(y)
        mlstm = case["mixer"] == "mlstm"
        states.append(_state_rows(carry["S"], carry["n"] if mlstm else None, carry["m"] if mlstm else None))
        if carry["kept"] is not None:
            kept.append(carry["kept"].reshape(-1))
    return {"out": torch.cat(ys), "state": ([torch.stack(kept)] if kept else []) + [torch.stack(states)]}


def _exact_experts(case, seed):
    rt = Runtime(torch.device("cuda", torch.cuda.current_device()), torch.bfloat16, PAGE)
    w = {k[2:]: v.double() for k, v in _weights(FEED_FORWARDS.build(_experts_spec(case), rt), seed, "l").items()}
    h = _rand(seed, "h", (case["tokens"], case["hidden"])).double()
    z = h @ w["router"].T
    top, idx = torch.topk(z, case["top"], dim=1)
    share = torch.softmax(top, dim=1)

    def unit(x, name):
        u = x @ w[name + ".up"].T
        if not case["gated"]:
            return torch.relu(u) ** 2 @ w[name + ".down"].T
        g = x @ w[name + ".gate"].T
        return (g * torch.sigmoid(g) * u) @ w[name + ".down"].T
    y = torch.zeros_like(h)
    for e in range(case["experts"]):
        row, col = torch.nonzero(idx == e, as_tuple=True)
        if row.numel():
            y.index_add_(0, row, share[row, col, None] * unit(h[row], f"e{e}"))
    if case["shared"] and case["gated"]:
        y += torch.sigmoid(h @ w["shared.sg"].T) * unit(h, "shared")
    return y
