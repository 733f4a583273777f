"""What a user of this framework has it do, as cases that can be measured.

Six kinds, each through entry points that a program can call:

    step       one step of a whole Qwen2-shaped model: `Engine.run_reserved` on a batch of single
               tokens and prompt portions, returning logits
    attention  a grouped-query attention mixer (q/k/v projection, rotation, cache write, paged
               attention, output projection) and the norm that adds its result to the stream
    mlp        a SwiGLU feed-forward and the norm behind it
    latent     a latent-attention mixer under a window with sinks, and the norm behind it
    moe        a routed mixture of experts and the norm behind it
    retention  a mixer with a matrix state per head, and the norm behind it

Sizes are the benchmark's three Qwen2.5 shapes and the layers that it puts at the same widths.
The layers of a step of single tokens are replayed from a CUDA graph, as the engine replays such a
step; prompt portions are launched one by one.
"""

from __future__ import annotations

import math

import torch

from somi_inference_b200.cache import CacheManager
from somi_inference_b200.config import Qwen2Config
from somi_inference_b200.config.spec import PartSpec
from somi_inference_b200.engine import Engine, StepEntry
from somi_inference_b200.engine.batch import BatchBuilder
from somi_inference_b200.ops import cuda_ops
from somi_inference_b200.parts import (FEED_FORWARDS, MIXERS, NORMS, BuildContext, declared_tensors)

SHAPES = {
    "0.5b": dict(layers=24, hidden=896, heads=14, kv_heads=2, dim=64, inter=4864, vocab=151936, tied=True,
                 eps=1e-6, q_rank=384, kv_rank=128),
    "7b": dict(layers=28, hidden=3584, heads=28, kv_heads=4, dim=128, inter=18944, vocab=152064, tied=False,
               eps=1e-6, q_rank=1536, kv_rank=512),
    "14b": dict(layers=48, hidden=5120, heads=40, kv_heads=8, dim=128, inter=13824, vocab=152064, tied=False,
                eps=1e-5, q_rank=1536, kv_rank=512),
}
THETA, PAGE, WINDOW, EXPERTS, TOP, GROUPS, KEEP = 1e6, 16, 1024, 16, 4, 4, 2
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    return [
        # a chat with one user on the smallest model: the shortest step there is
        dict(name="step-0.5b-one-token", kind="step", shape="0.5b", layers=24, dtype="bfloat16",
             decode=1, context=130, portion=0, portion_context=0),
        # the command line's and LLM's default type: a short prompt beside a few running requests
        dict(name="step-0.5b-float32-mixed", kind="step", shape="0.5b", layers=24, dtype="float32",
             decode=4, context=300, portion=203, portion_context=0),
        # the benchmark's headline step: 8 requests at 2,048 cached tokens
        dict(name="attention-7b-decode-8", kind="attention", shape="7b", dtype="bfloat16",
             decode=8, context=2048, portion=0, portion_context=0),
        # a loaded server: 64 requests of unequal lengths
        dict(name="attention-14b-decode-64", kind="attention", shape="14b", dtype="bfloat16",
             decode=64, context=4001, portion=0, portion_context=0),
        # the benchmark's prompt
        dict(name="attention-7b-prompt-2048", kind="attention", shape="7b", dtype="bfloat16",
             decode=0, context=0, portion=2048, portion_context=0),
        # a long prompt on the small model, whose head size is 64; no multiple of any tile
        dict(name="attention-0.5b-prompt-8111", kind="attention", shape="0.5b", dtype="bfloat16",
             decode=0, context=0, portion=8111, portion_context=0),
        # decoding in the default type
        dict(name="attention-0.5b-float32-decode-4", kind="attention", shape="0.5b", dtype="float32",
             decode=4, context=1000, portion=0, portion_context=0),
        # the headline step's feed-forward, where most of its bytes are
        dict(name="mlp-7b-8", kind="mlp", shape="7b", dtype="bfloat16", tokens=8),
        # a prompt's feed-forward, where most of its operations are
        dict(name="mlp-7b-1999", kind="mlp", shape="7b", dtype="bfloat16", tokens=1999),
        # a prompt through a layer that caches a latent
        dict(name="latent-7b-prompt-2048", kind="latent", shape="7b", dtype="bfloat16",
             decode=0, context=0, portion=2048, portion_context=0),
        # the headline step on a layer of experts
        dict(name="moe-7b-8", kind="moe", shape="7b", dtype="bfloat16", tokens=8),
        # a prompt through a layer that carries a state
        dict(name="retention-7b-prompt-2048", kind="retention", shape="7b", dtype="bfloat16",
             decode=0, context=0, portion=2048, portion_context=0),
    ]


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


def _draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))

    def requests():
        """Single tokens, a portion of a prompt (from its start or behind earlier ones), or both."""
        what = rng.choice(("decode", "decode", "portion", "portion", "both"))
        d, c, p, pc = 0, 0, 0, 0
        if what != "portion":
            d, c = size(1, 64), size(16, 8192)
        if what != "decode":
            p, pc = size(2, 8192 if what == "portion" else 1024), rng.choice((0, 0, size(16, 4096)))
        return dict(decode=d, context=c, portion=p, portion_context=pc)

    kind = rng.choice(("step", "attention", "attention", "attention", "mlp", "mlp", "latent", "moe", "retention"))
    dtype = rng.choice(("bfloat16", "bfloat16", "bfloat16", "float32"))
    if kind == "step":
        return dict(kind=kind, shape="0.5b", layers=24, dtype=dtype, decode=size(1, 16), context=size(16, 600),
                    portion=rng.choice((0, size(2, 300))), portion_context=0)
    shape = "0.5b" if dtype == "float32" else rng.choice(("0.5b", "7b", "14b") if kind in ("attention", "mlp")
                                                         else ("0.5b", "7b"))
    if kind in ("mlp", "moe"):
        return dict(kind=kind, shape=shape, dtype=dtype, tokens=size(1, 4096))
    case = dict(kind=kind, shape=shape, dtype=dtype, **requests())
    if kind == "retention":
        case["portion_context"] = 0          # (a state is all that is left of earlier portions)
    return case


# ------------------------------------------------------------------------------------ requests
def _contexts(case):
    """Cached tokens of the single-token requests: unequal, from half of `context` up to it."""
    c = case["context"]
    return [c - (97 * i) % max(1, c // 2) for i in range(case["decode"])]


def _requests(case):
    """(cached tokens, tokens in this step) per request; the prompt portion comes first."""
    head = [(case["portion_context"], case["portion"])] if case["portion"] else []
    return head + [(c, 1) for c in _contexts(case)]


def _tokens(case):
    return case["tokens"] if "tokens" in case else sum(q for _, q in _requests(case))


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * stream + seed)


def _normal(gen, shape, std, dtype):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, std, generator=gen).to(dtype)


# ------------------------------------------------------------------------------------ weights
def _part(case):
    """The case's part as the framework's registries take it."""
    s = SHAPES[case["shape"]]
    D, H, d, inter = s["hidden"], s["heads"], s["dim"], s["inter"]
    if case["kind"] == "attention":
        names = {f"{p}_{w}": f"{p}.{w}" for p in "qkv" for w in ("weight", "bias")}
        return PartSpec("attention", {
            "hidden_size": D, "num_heads": H, "num_kv_heads": s["kv_heads"], "head_dim": d, "qkv_bias": True,
            "out_bias": False, "window": None,
            "position": PartSpec("rope", {"head_dim": d, "theta": THETA, "max_positions": 40960}),
            "names": {**names, "o_weight": "o.weight"}})
    if case["kind"] == "mlp":
        return PartSpec("swiglu", {"hidden_size": D, "intermediate_size": inter,
                                   "names": {"gate_weight": "gate", "up_weight": "up", "down_weight": "down"}})
    if case["kind"] == "latent":
        names = ("q_down", "q_norm", "q_up", "k_up", "v_up", "sink", "out", "kv_down", "kv_norm")
        return PartSpec("latent_attention", {
            "hidden_size": D, "heads": H, "key_dim": d, "value_dim": d, "q_rank": s["q_rank"],
            "kv_rank": s["kv_rank"], "scale": d ** -0.5, "window": WINDOW, "own_latent": True, "sink": True,
            "eps": s["eps"], "names": {n: n for n in names}})
    if case["kind"] == "moe":
        return PartSpec("routed_moe", {
            "hidden_size": D, "experts": EXPERTS, "top": TOP, "expert_ff": inter // 4, "scores": "sigmoid",
            "correction": True, "groups": {"count": GROUPS, "keep": KEEP, "best": 2},
            "names": {"router": "router", "correction": "correction",
                      **{p: [f"{p}.{e}" for e in range(EXPERTS)] for p in ("gate", "up", "down")}}})
    names = {f"{p}_weight": p for p in ("q", "k", "v", "o", "gate")}
    return PartSpec("retention", {
        "hidden_size": D, "heads": H, "key_dim": d, "value_dim": d, "decay": _decays(H),
        "rotary": {"dims": d, "base": THETA}, "k_scale": d ** -0.5, "eps": s["eps"], "names": names})


def _decays(heads):
    return [1.0 - 2.0 ** -(5.0 + 7.0 * h / max(1, heads - 1)) for h in range(heads)]


def _weights(case, decls, seed):
    """Seeded weights in the case's type: matrices and biases N(0, 0.02), norm weights about 1."""
    gen, dtype, out = _generator(seed, 1), DTYPES[case["dtype"]], {}
    for d in sorted(decls, key=lambda t: t.name):
        if d.ignored:
            continue
        t = _normal(gen, d.shape, 0.02, dtype)
        out[d.name] = (1.0 + 5.0 * t.float()).to(dtype) if d.init == "ones" else t
    return out


def _layer_inputs(case, seed):
    """Normed rows, the residual stream and the weight of the norm behind the part."""
    s, gen, T = SHAPES[case["shape"]], _generator(seed, 2), _tokens(case)
    x = _normal(gen, (T, s["hidden"]), 1.0, DTYPES[case["dtype"]])
    residual = _normal(gen, (T, s["hidden"]), 0.1, torch.float32)
    weight = (1.0 + _normal(gen, (s["hidden"],), 0.1, torch.float32)).to(DTYPES[case["dtype"]])
    return x, residual, weight


def _cached_rows(case, seed):
    """Per request what earlier steps left in its cache: keys and values, or latents."""
    s, gen, dtype = SHAPES[case["shape"]], _generator(seed, 3), DTYPES[case["dtype"]]
    if case["kind"] == "attention":
        shape = (s["kv_heads"], s["dim"])
        return [(_normal(gen, (c, *shape), 1.2, dtype), _normal(gen, (c, *shape), 1.2, dtype))
                for c, _ in _requests(case)]
    return [(_normal(gen, (c, 1, s["kv_rank"]), 1.0, dtype),) for c, _ in _requests(case)]


def _first_states(case, seed):
    """The states that the requests' earlier tokens left (zeros before a prompt's first token)."""
    s, gen = SHAPES[case["shape"]], _generator(seed, 3)
    states = _normal(gen, (len(_requests(case)), s["heads"], s["dim"], s["dim"]), 3.0, torch.float32)
    if case["portion"]:
        states[0] = 0.0
    return states


def _step_config(case):
    s = SHAPES[case["shape"]]
    return Qwen2Config.from_dict(dict(
        num_hidden_layers=case["layers"], hidden_size=s["hidden"], num_attention_heads=s["heads"],
        num_key_value_heads=s["kv_heads"], head_dim=s["dim"], intermediate_size=s["inter"],
        vocab_size=s["vocab"], rope_theta=THETA, rms_norm_eps=s["eps"], tie_word_embeddings=s["tied"],
        max_position_embeddings=4096, architectures=["Qwen2ForCausalLM"], hidden_act="silu",
        use_sliding_window=False))


def _step_tokens(case, seed):
    """All token ids of each request, those that earlier steps ran first."""
    gen = _generator(seed, 2)
    return [torch.randint(0, SHAPES[case["shape"]]["vocab"], (c + q,), generator=gen, device="cuda").tolist()
            for c, q in _requests(case)]


# ------------------------------------------------------------------------------------ prepare and run
class _State:
    """What a program keeps between calls: `call()` makes one pass; `held` is what that reads (a
    replayed graph knows addresses only)."""

    def __init__(self, call, *held):
        self.call, self.held = call, held


def prepare(case, seed):
    with torch.no_grad():
        return _prepare_step(case, seed) if case["kind"] == "step" else _prepare_layer(case, seed)


def run(state):
    with torch.no_grad():
        return state.call()


def _prepare_step(case, seed):
    cfg, reqs = _step_config(case), _requests(case)
    weights = _weights(case, declared_tensors(cfg.to_model_spec()).values(), seed)
    engine = Engine.from_tensors(cfg, weights, dtype=case["dtype"], page_size=PAGE, max_requests=len(reqs),
                                 max_tokens=sum(c + q + PAGE for c, q in reqs))
    entries = []
    for i, ((c, q), ids) in enumerate(zip(reqs, _step_tokens(case, seed))):
        if c:
            engine.step([StepEntry(i, ids[:c], [])])
        else:
            engine.cache.register(i)
        engine.cache.reserve(i, q)
        entries.append(StepEntry(i, ids[c:], [q - 1]))
    return _State(lambda: engine.run_reserved(entries), engine)


def _prepare_layer(case, seed):
    dtype, device = DTYPES[case["dtype"]], torch.device("cuda", torch.cuda.current_device())
    ctx = BuildContext(dtype=dtype, device=device, ops=cuda_ops())
    spec, s = _part(case), SHAPES[case["shape"]]
    registry = FEED_FORWARDS if case["kind"] in ("mlp", "moe") else MIXERS
    decls = registry.declare(spec)
    weights = _weights(case, decls, seed)
    part = registry.build(spec, {d.name: ctx.place(weights[d.name], matrix=d.matrix) for d in decls}, ctx)
    del weights
    x, residual, weight = _layer_inputs(case, seed)
    norm = NORMS.build(PartSpec("rmsnorm", {"size": s["hidden"], "eps": s["eps"], "names": {"weight": "w"}}),
                       {"w": weight}, ctx)
    rows = torch.arange(x.shape[0], dtype=torch.int32, device=device)      # (the stream itself stays as it is)
    if registry is FEED_FORWARDS:
        def layer():
            return norm.forward(residual, part.forward(x, None), rows)
        return _State(_captured(layer) if x.shape[0] <= 64 else layer, layer)

    reqs = _requests(case)
    blocks = [-(-(c + q) // PAGE) for c, q in reqs]
    mgr = CacheManager([part.cache_needs()], [None], num_pages=sum(blocks) + 1, page_size=PAGE,
                       max_requests=len(reqs), max_positions=max(c + q for c, q in reqs) + PAGE,
                       dtype=dtype, device=device)
    for group in mgr.groups:                  # as after a while of serving: pages in no order
        taken = group.pool.take(group.pool.num_free)
        order = torch.randperm(len(taken), generator=torch.Generator().manual_seed(seed)).tolist()
        group.pool.give_back([taken[i] for i in order])
    entries = []
    for i, (c, q) in enumerate(reqs):
        mgr.register(i)
        if c:
            mgr.reserve(i, c)
            mgr.commit(i)
        mgr.reserve(i, q)
        entries.append(StepEntry(i, [0] * q, []))
    builder = BatchBuilder(mgr, device=device, q_tile_sizes=ctx.ops.q_tile_sizes)
    batch, _ = builder.build(entries)
    view = mgr.view(0)
    if case["kind"] == "retention":
        slots = batch.state_slot.long()
        (state,) = view.state.values()
        start = torch.zeros_like(state)
        start[slots] = _first_states(case, seed).transpose(2, 3)

        def layer():
            state.copy_(start)                # where the request was before this step
            return {"out": norm.forward(residual, part.forward(x, batch, view, True), rows),
                    "state": state[slots]}
        return _State(_captured(layer) if not case["portion"] else layer, layer, builder)
    for i, cached in enumerate(_cached_rows(case, seed)):
        # (positions that a window has passed have no page any more)
        pos = torch.arange(cached[0].shape[0], device=device)
        page = batch.groups[0].block_table[i].long()[pos // PAGE]
        pos, page = pos[page >= 0], page[page >= 0]
        for store, kept in zip((view.paged.keys, view.paged.values), cached):
            store[page, :, pos % PAGE] = kept[pos]

    def layer():
        return norm.forward(residual, part.forward(x, batch, view, True), rows)
    return _State(_captured(layer) if not case["portion"] else layer, layer, builder)


def _captured(layer):
    layer()
    layer()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = layer()

    def replay():
        graph.replay()
        return out
    return replay


# ------------------------------------------------------------------------------------ work and tolerance
def _pairs(case, window=None):
    """(query, key) pairs that the mask leaves, and cached or new rows that some query reads."""
    pairs = rows = 0
    for c, q in _requests(case):
        w = window or c + q
        n = min(q, max(0, w - c))             # queries that still see everything
        pairs += n * c + n * (n + 1) // 2 + (q - n) * w
        rows += min(c + q, w + q - 1)
    return pairs, rows


def work(case):
    s, T = SHAPES[case["shape"]], _tokens(case)
    b = 2 if case["dtype"] == "bfloat16" else 4
    D, H, G, d, inter = s["hidden"], s["heads"], s["kv_heads"], s["dim"], s["inter"]
    ends = T * D * (b + 4 + b)                # the part's input, the stream, the normed result
    qkvo = D * (H + 2 * G) * d + H * d * D
    if case["kind"] == "step":
        layer, wanted = qkvo + 3 * D * inter, len(_requests(case))
        pairs, rows = _pairs(case)
        L = case["layers"]
        return {"bytes": b * (L * layer + s["vocab"] * D) + L * rows * 2 * G * d * b + wanted * s["vocab"] * 4,
                "flops": 2.0 * T * L * layer + 2.0 * wanted * s["vocab"] * D + 4.0 * L * H * d * pairs}
    if case["kind"] == "attention":
        pairs, rows = _pairs(case)
        return {"bytes": ends + qkvo * b + rows * 2 * G * d * b + T * 2 * G * d * b,
                "flops": 2.0 * T * qkvo + 4.0 * H * d * pairs}
    if case["kind"] == "mlp":
        return {"bytes": ends + 3 * D * inter * b, "flops": 6.0 * T * D * inter}
    if case["kind"] == "latent":
        # the way that needs the fewest operations: keys and values expanded once for a portion, or
        # the expansions on the query side and behind the sum for a single token
        rq, rk = s["q_rank"], s["kv_rank"]
        base = D * (rq + rk) + rq * H * d + H * d * D
        pairs, rows = _pairs(case, WINDOW)
        expanded = 2.0 * rows * rk * 2 * H * d + 4.0 * H * d * pairs
        absorbed = 4.0 * T * H * d * rk + 4.0 * H * rk * pairs
        return {"bytes": ends + (base + 2 * rk * H * d) * b + (rows + T) * rk * b,
                "flops": 2.0 * T * base + min(expanded, absorbed)}
    if case["kind"] == "moe":
        ff = inter // 4
        hit = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** T)        # experts that some token chooses
        return {"bytes": ends + D * EXPERTS * b + hit * 3 * D * ff * b,
                "flops": 2.0 * T * D * EXPERTS + 6.0 * T * TOP * D * ff}
    R = len(_requests(case))
    return {"bytes": ends + 5 * D * H * d * b + 2 * R * H * d * d * 4,
            "flops": 2.0 * T * 5 * D * H * d + 5.0 * T * H * d * d}


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (1.6e15 if case["dtype"] == "bfloat16" else 6e13))


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "step":
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.2}


# ------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return _exact_step(case, seed) if case["kind"] == "step" else _exact_layer(case, seed)


def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight.double()


def _turn(x, pos, d):
    """Entry i < d / 2 of every head [T, heads, d] paired with entry i + d / 2 and turned."""
    freq = THETA ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    angle = pos.double()[:, None, None] * freq
    c, s, a, b = torch.cos(angle), torch.sin(angle), x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, first, scale, window=None, sink=None):
    """Causal attention of rows q [T, H, d] at positions first.. over k, v [S, G, *] from position 0."""
    T, H, S = q.shape[0], q.shape[1], k.shape[0]
    out = torch.empty((T, H, v.shape[2]), dtype=torch.float64, device=q.device)
    key = torch.arange(S, device=q.device)
    step = max(1, (1 << 26) // S)
    for h in range(H):
        g = h // (H // k.shape[1])
        for lo in range(0, T, step):
            pos = first + torch.arange(lo, min(T, lo + step), device=q.device)[:, None]
            s = (q[lo:lo + step, h] @ k[:, g].T) * scale
            hidden = key > pos if window is None else (key > pos) | (key <= pos - window)
            s.masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
            out[lo:lo + step, h] = torch.softmax(s, 1)[:, :S] @ v[:, g]
    return out


def _swiglu(x, gate, up, down):
    return (torch.nn.functional.silu(x @ gate.double().T) * (x @ up.double().T)) @ down.double().T


def _exact_step(case, seed):
    s, cfg = SHAPES[case["shape"]], _step_config(case)
    w = _weights(case, declared_tensors(cfg.to_model_spec()).values(), seed)
    D, H, G, d, eps = s["hidden"], s["heads"], s["kv_heads"], s["dim"], s["eps"]
    ids = _step_tokens(case, seed)
    cuts = [0]
    for t in ids:
        cuts.append(cuts[-1] + len(t))
    x = w["model.embed_tokens.weight"][torch.tensor(sum(ids, []), device="cuda")].double()
    pos = torch.cat([torch.arange(len(t), device="cuda") for t in ids])
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps, w[p + "input_layernorm.weight"])
        q, k, v = (h @ w[f"{p}self_attn.{n}_proj.weight"].double().T + w[f"{p}self_attn.{n}_proj.bias"].double()
                   for n in "qkv")
        q, k, v = _turn(q.view(-1, H, d), pos, d), _turn(k.view(-1, G, d), pos, d), v.view(-1, G, d)
        a = torch.cat([_attend(q[lo:hi], k[lo:hi], v[lo:hi], 0, d ** -0.5) for lo, hi in zip(cuts, cuts[1:])])
        x = x + a.reshape(-1, H * d) @ w[p + "self_attn.o_proj.weight"].double().T
        h = _rms(x, eps, w[p + "post_attention_layernorm.weight"])
        x = x + _swiglu(h, *(w[f"{p}mlp.{n}_proj.weight"] for n in ("gate", "up", "down")))
    h = _rms(x[[c - 1 for c in cuts[1:]]], eps, w["model.norm.weight"])
    return h @ w["model.embed_tokens.weight" if s["tied"] else "lm_head.weight"].double().T


def _exact_layer(case, seed):
    s, spec = SHAPES[case["shape"]], _part(case)
    decls = (FEED_FORWARDS if case["kind"] in ("mlp", "moe") else MIXERS).declare(spec)
    w = _weights(case, decls, seed)
    x, residual, weight = _layer_inputs(case, seed)
    y = {"attention": _exact_attention, "mlp": _exact_mlp, "latent": _exact_latent, "moe": _exact_moe,
         "retention": _exact_retention}[case["kind"]](case, seed, s, w, x.double())
    state = None
    if case["kind"] == "retention":
        y, state = y
    out = _rms(residual.double() + y, s["eps"], weight)
    return out if state is None else {"out": out, "state": state}


def _exact_attention(case, seed, s, w, x):
    H, G, d = s["heads"], s["kv_heads"], s["dim"]
    q, k, v = ((x @ w[f"{n}.weight"].double().T + w[f"{n}.bias"].double()).view(x.shape[0], -1, d) for n in "qkv")
    out, row = [], 0
    for (c, n), (kc, vc) in zip(_requests(case), _cached_rows(case, seed)):
        pos, at = c + torch.arange(n, device="cuda"), slice(row, row + n)
        keys = torch.cat([kc.double(), _turn(k[at], pos, d)])
        out.append(_attend(_turn(q[at], pos, d), keys, torch.cat([vc.double(), v[at]]), c, d ** -0.5))
        row += n
    return torch.cat(out).reshape(-1, H * d) @ w["o.weight"].double().T


def _exact_mlp(case, seed, s, w, x):
    return _swiglu(x, w["gate"], w["up"], w["down"])


def _exact_latent(case, seed, s, w, x):
    H, d, r = s["heads"], s["dim"], s["kv_rank"]
    q = _rms(x @ w["q_down"].double().T, s["eps"], w["q_norm"]) @ w["q_up"].double().T
    new = _rms(x @ w["kv_down"].double().T, s["eps"], w["kv_norm"])
    out, row = [], 0
    for (c, n), (cached,) in zip(_requests(case), _cached_rows(case, seed)):
        lat = torch.cat([cached.double().view(c, r), new[row:row + n]])
        keys, values = ((lat @ w[m].double().T).view(-1, H, d) for m in ("k_up", "v_up"))
        out.append(_attend(q[row:row + n].view(n, H, d), keys, values, c, d ** -0.5, WINDOW, w["sink"].double()))
        row += n
    return torch.cat(out).reshape(-1, H * d) @ w["out"].double().T


def _exact_moe(case, seed, s, w, x):
    score = torch.sigmoid(x @ w["router"].double().T)
    choice = (score + w["correction"].double()).view(-1, GROUPS, EXPERTS // GROUPS)
    best = choice.topk(2, -1).values.sum(-1).topk(KEEP, -1).indices
    kept = torch.zeros(choice.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, best, True)
    chosen = choice.masked_fill(~kept[..., None], -math.inf).flatten(1).topk(TOP, -1).indices
    y = torch.zeros_like(x)
    for e in range(EXPERTS):
        rows = (chosen == e).any(1).nonzero()[:, 0]
        y[rows] += score[rows, e, None] * _swiglu(x[rows], w[f"gate.{e}"], w[f"up.{e}"], w[f"down.{e}"])
    return y


def _exact_retention(case, seed, s, w, x):
    H, d = s["heads"], s["dim"]
    q, k, v, z = ((x @ w[n].double().T).view(-1, H, d) for n in ("q", "k", "v", "gate"))
    decay = torch.tensor(_decays(H), dtype=torch.float64, device="cuda")[:, None, None]
    states, out, row = _first_states(case, seed).double(), torch.empty_like(q), 0
    for r, (c, n) in enumerate(_requests(case)):
        at = slice(row, row + n)
        pos = c + torch.arange(n, device="cuda")
        # (the state holds what the keys wrote without their factor, which the queries carry)
        qt, kt, vt, m = _turn(q[at], pos, d) * d ** -0.5, _turn(k[at], pos, d), v[at], states[r]
        for t in range(n):
            m = decay * m + kt[t][:, :, None] * vt[t][:, None, :]
            out[row + t] = (qt[t][:, None, :] @ m)[:, 0]
        states[r] = m
        row += n
    o = _rms(out, s["eps"]) * torch.nn.functional.silu(z)
    return o.reshape(-1, H * d) @ w["o"].double().T, states.transpose(2, 3)
