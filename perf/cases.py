"""The work that a user has this framework do, as cases that can be timed and checked: whole steps of a Llama-shaped
model through `Engine`, and single layers through the parts and operators that models are put together from.

The sizes are those of the benchmark (the 1B Llama shape), of the designs' configurations at widths 2,048 and 4,096, and
ragged lengths between.  `listed()` gives the named cases, `draw(rng)` one more of the same ranges; `prepare` makes a
case's inputs and handles on the device, `run` is one pass, `exact` the same results in plain torch at 64 bits."""
from __future__ import annotations

import math

import torch

from picolm_b200 import ops
from picolm_b200.cache import SequenceCache
from picolm_b200.cache.sequence_cache import KVLayerCache, StateLayerCache
from picolm_b200.cache.spec import CacheSpec
from picolm_b200.config.registry import config_from_dict, spec_of
from picolm_b200.config.spec import PartSpec
from picolm_b200.engine.engine import Engine
from picolm_b200.engine.model import Model
from picolm_b200.engine.step_batch import build_step_batch
from picolm_b200.parts import build_part
from picolm_b200.runtime import Runtime

DEVICE = "cuda:0"
LLAMA_1B = dict(layers=16, width=2048, ff=8192, heads=32, kv_heads=8, head_dim=64, vocab=128256)
LLAMA_W2048 = dict(width=2048, ff=8192, heads=32, kv_heads=8, head_dim=64, vocab=32000)
LLAMA_W4096 = dict(width=4096, ff=14336, heads=32, kv_heads=8, head_dim=128, vocab=32000)
ROPE_THETA = 500000.0
EPS = 1e-5
STD = 0.02                       # of a random matrix


def listed():
    return [
        # A prompt of a chat or a document, read in one step, its last token's logits wanted: the benchmark's prompt.
        dict(name="prompt", kind="llama", dtype="bfloat16", seqs=1, prompt=2048, new=0, want="last", **LLAMA_1B),
        # Eight requests served together: prompts of unequal lengths, then single-token steps, the benchmark's decode.
        dict(name="generate", kind="llama", dtype="bfloat16", seqs=8, prompt=1024, new=64, want="last", **LLAMA_1B),
        # The 32-bit run that results are checked against (trace replay): every token's logits, an odd number of tokens.
        dict(name="prompt float32", kind="llama", dtype="float32", seqs=2, prompt=301, new=0, want="all", layers=2, **LLAMA_W2048),
        # Attention of prompts in a batch: unequal lengths, heads of 128 in groups of four.
        dict(name="attention prompt", kind="attention", heads=32, kv_heads=8, head_dim=128, seqs=3, new=4096, context=0, window=0),
        # Attention of a large batch's single-token step over unequal contexts.
        dict(name="attention decode", kind="attention", heads=32, kv_heads=8, head_dim=64, seqs=64, new=1, context=4096, window=0),
        # The feed-forward of a wide model on a prompt of an odd length.
        dict(name="mlp prompt", kind="mlp", width=4096, ff=14336, tokens=1500),
        # The same for the few tokens of a small batch's single-token step.
        dict(name="mlp few", kind="mlp", width=4096, ff=14336, tokens=5),
        # Routed experts with a shared one on a prompt.
        dict(name="routed prompt", kind="routed", width=2048, ff=2048, experts=32, top=3, groups=4, shared=2048, gated=True, tokens=2048),
        # Routed experts without a gate on a single-token step of eight sequences.
        dict(name="routed few", kind="routed", width=4096, ff=5376, experts=16, top=4, groups=1, shared=0, gated=False, tokens=8),
        # Recurrent mixers on prompts: a delta rule with a decay per key channel, ...
        dict(name="delta prompt", kind="delta", width=2048, heads=8, kv_heads=4, dim=128, vdim=128, decay="channel", seqs=1, tokens=2048),
        # ... linear attention with a learned decay per key channel, ...
        dict(name="gla prompt", kind="gla", width=2048, heads=8, dim=128, vdim=256, seqs=2, tokens=1537),
        # ... and retention, a constant decay a head over rotated queries and keys.
        dict(name="retention prompt", kind="retention", width=4096, heads=16, dim=128, vdim=256, seqs=1, tokens=2048),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, evenly over its logarithm; odd ones as often as even ones."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["prompt", "generate", "float32", "attention prompt", "attention decode", "mlp prompt", "mlp few",
                       "routed prompt", "routed few", "delta", "gla", "retention"])
    if what in ("prompt", "generate", "float32"):
        shape = rng.choice([LLAMA_W2048, LLAMA_W4096])
        if what == "prompt":
            return dict(kind="llama", dtype="bfloat16", seqs=rng.randint(1, 3), prompt=_log(rng, 64, 2048), new=0, want="last",
                        layers=rng.randint(2, 4), **shape)
        if what == "generate":
            return dict(kind="llama", dtype="bfloat16", seqs=_log(rng, 1, 24), prompt=_log(rng, 16, 512), new=rng.randint(16, 48),
                        want="last", layers=rng.randint(2, 4), **shape)
        return dict(kind="llama", dtype="float32", seqs=rng.randint(1, 3), prompt=_log(rng, 24, 400), new=0, want="all", layers=1,
                    **shape)
    if what.startswith("attention"):
        heads = dict(kv_heads=8, head_dim=rng.choice([64, 128]), heads=rng.choice([16, 32]))
        if what == "attention prompt":
            return dict(kind="attention", seqs=rng.randint(1, 4), new=_log(rng, 100, 4096), context=rng.choice([0, 0, 1000]),
                        window=rng.choice([0, 0, 0, 1024]), **heads)
        return dict(kind="attention", seqs=_log(rng, 4, 96), new=1, context=_log(rng, 500, 6000), window=0, **heads)
    width, ff = rng.choice([(2048, 8192), (4096, 14336)])
    if what == "mlp prompt":
        return dict(kind="mlp", width=width, ff=ff, tokens=_log(rng, 65, 3000))
    if what == "mlp few":
        return dict(kind="mlp", width=width, ff=ff, tokens=_log(rng, 1, 64))
    if what.startswith("routed"):
        gated = rng.random() < 0.5
        return dict(kind="routed", width=width, ff=ff // 4 if gated else 3 * ff // 8, experts=32 if width == 2048 else 16,
                    top=rng.randint(2, 4), groups=rng.choice([1, 4]), shared=rng.choice([0, ff // 4]) if gated else 0, gated=gated,
                    tokens=_log(rng, 256, 3000) if what == "routed prompt" else _log(rng, 1, 48))
    heads = width // 256
    lengths = dict(seqs=rng.randint(1, 4), tokens=_log(rng, 100, 2048))
    if what == "delta":
        return dict(kind="delta", width=width, heads=heads, kv_heads=rng.choice([heads, heads // 2]), dim=rng.choice([64, 128]), vdim=128,
                    decay=rng.choice(["channel", "channel", "head"]), **lengths)
    if what == "gla":
        return dict(kind="gla", width=width, heads=heads, dim=rng.choice([64, 128]), vdim=rng.choice([128, 256]), **lengths)
    return dict(kind="retention", width=width, heads=heads, dim=rng.choice([64, 128]), vdim=rng.choice([128, 256]), **lengths)


# ------------------------------------------------------------------------------------------------- inputs
def _lengths(n, longest):
    """n unequal lengths, the first the longest, the others down to a quarter of it."""
    return [max(1, int(longest * (1.0 - 0.75 * ((i * 0.6180339887) % 1.0)))) for i in range(n)]


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _normal(shape, g, scale=1.0, dtype=torch.bfloat16):
    """Normal numbers times `scale`, rounded to bfloat16 whatever type they are kept in."""
    return (torch.randn(shape, generator=g, device=DEVICE) * scale).to(torch.bfloat16).to(dtype)


def _tensors(specs, g, dtype=torch.bfloat16):
    out = {}
    for name in sorted(specs):
        ws = specs[name]
        if ws.init == "uniform":
            t = ws.lo + (ws.hi - ws.lo) * torch.rand(ws.shape, generator=g, device=DEVICE)
        elif ws.init == "ones_normal":
            t = 1.0 + 0.1 * torch.randn(ws.shape, generator=g, device=DEVICE)
        else:
            t = torch.randn(ws.shape, generator=g, device=DEVICE) * (ws.scale if ws.init == "normal_scaled" else STD)
        out[name] = t.to(torch.bfloat16).to(dtype)
    return out


def _type(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


# --------------------------------------------------------------------------------------- whole model steps
_engine = [None, None]          # what a server keeps: the engine of one model, loaded once


def _llama_model(case, runtime):
    cfg = config_from_dict({
        "architectures": ["LlamaForCausalLM"], "vocab_size": case["vocab"], "hidden_size": case["width"],
        "intermediate_size": case["ff"], "num_hidden_layers": case["layers"], "num_attention_heads": case["heads"],
        "num_key_value_heads": case["kv_heads"], "head_dim": case["head_dim"], "rms_norm_eps": EPS, "rope_theta": ROPE_THETA,
        "max_position_embeddings": 8192, "tie_word_embeddings": True})
    return Model(spec_of(cfg), runtime)


def _llama_engine(case):
    lengths = [n + case["new"] for n in _lengths(case["seqs"], case["prompt"])]
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _engine[0] != key:
        _engine[:] = [None, None]
        model = _llama_model(case, Runtime.create(case["dtype"], DEVICE))
        tensors = _tensors(model.expected_tensors(), _generator(7), _type(case))
        model.load_tensors(lambda name: tensors[name])
        room = sum((n + 63) // 64 * 64 for n in lengths)
        _engine[:] = [key, Engine(model, max_tokens=room, max_seqs=case["seqs"], max_seq_tokens=max(lengths))]
    return _engine[1]


def _llama_tokens(case, seed):
    """Each sequence's prompt and the tokens that it goes on with."""
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, case["vocab"], (n + case["new"],), generator=g).tolist() for n in _lengths(case["seqs"], case["prompt"])]


def _prepare_llama(case, seed):
    rows = _llama_tokens(case, seed)
    lens = _lengths(case["seqs"], case["prompt"])
    prompts = [r[:n] for r, n in zip(rows, lens)]
    steps = [[r[n + i] for r, n in zip(rows, lens)] for i in range(case["new"])]
    out = None
    if steps:
        out = torch.empty((case["new"] + 1, case["seqs"], case["vocab"]), device=DEVICE)
    wants = [list(range(n)) for n in lens] if case["want"] == "all" else None
    return dict(kind="llama", engine=_llama_engine(case), prompts=prompts, steps=steps, wants=wants, out=out)


def _run_llama(s):
    eng = s["engine"]
    slots = [eng.new_sequence() for _ in s["prompts"]]
    try:
        logits = eng.step(list(zip(slots, s["prompts"])), s["wants"])
        if s["out"] is None:
            return logits.clone()
        s["out"][0].copy_(logits)
        for i, tokens in enumerate(s["steps"]):
            s["out"][i + 1].copy_(eng.step([(slot, [t]) for slot, t in zip(slots, tokens)]))
        return s["out"]
    finally:
        for slot in slots:
            eng.end_sequence(slot)


def _exact_llama(case, seed):
    model = _llama_model(case, None)
    w = _tensors(model.expected_tensors(), _generator(7), _type(case))
    rows, lens = _llama_tokens(case, seed), _lengths(case["seqs"], case["prompt"])
    H, G, hd = case["heads"], case["kv_heads"], case["head_dim"]
    freq = ROPE_THETA ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=DEVICE) / hd)

    def norm(x, name):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w[name].double()

    def rotate(x):                                               # [n, heads, hd], halves paired
        angle = torch.arange(x.shape[0], dtype=torch.float64, device=DEVICE)[:, None] * freq
        c, s = angle.cos()[:, None], angle.sin()[:, None]
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    xs = [w["model.embed_tokens.weight"][torch.tensor(r, device=DEVICE)].double() for r in rows]
    for i in range(case["layers"]):
        at = f"model.layers.{i}."
        m = {k: w[at + k + ".weight"].double() for k in ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
                                                        "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        for b, x in enumerate(xs):
            n = x.shape[0]
            h = norm(x, at + "input_layernorm.weight")
            q = rotate((h @ m["self_attn.q_proj"].T).view(n, H, hd))
            k = rotate((h @ m["self_attn.k_proj"].T).view(n, G, hd))
            v = (h @ m["self_attn.v_proj"].T).view(n, G, hd)
            x = x + _attend(q, k, v, 0, hd ** -0.5, 0) @ m["self_attn.o_proj"].T
            h = norm(x, at + "post_attention_layernorm.weight")
            xs[b] = x + (torch.nn.functional.silu(h @ m["mlp.gate_proj"].T) * (h @ m["mlp.up_proj"].T)) @ m["mlp.down_proj"].T
        del m
    if case["want"] == "all":
        picked = torch.cat(xs)
    else:
        picked = torch.stack([x[n - 1 + i] for i in range(case["new"] + 1) for x, n in zip(xs, lens)])
    h = norm(picked, "model.norm.weight")
    head = w["model.embed_tokens.weight"]
    logits = torch.cat([h @ head[a:a + 16384].double().T for a in range(0, case["vocab"], 16384)], 1)
    return logits.view(case["new"] + 1, case["seqs"], -1) if case["new"] else logits


# ------------------------------------------------------------------------------------------------ attention
def _attend(q, k, v, first, scale, window):
    """Causal attention of q [n, H, hd], the first row at position `first`, over k, v [m, G, hd]; [n, H * hd]."""
    n, H, hd = q.shape
    m, G = k.shape[:2]
    at = first + torch.arange(n, device=q.device)[:, None]
    key = torch.arange(m, device=q.device)[None]
    hidden = (key > at) | (key <= at - window if window else torch.zeros_like(key, dtype=torch.bool))
    out = torch.empty((n, H, hd), dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        out[:, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:, h // (H // G)]
    return out.reshape(n, H * hd)


def _attention_lengths(case):
    """(positions already in the cache, new ones) of each sequence."""
    if case["new"] == 1:
        return [(n, 1) for n in _lengths(case["seqs"], case["context"])]
    return [(case["context"] // (1 + b), n) for b, n in enumerate(_lengths(case["seqs"], case["new"]))]


def _attention_inputs(case, seed):
    g = _generator(seed)
    H, G, hd = case["heads"], case["kv_heads"], case["head_dim"]
    lens = _attention_lengths(case)
    q = _normal((sum(n for _, n in lens), H, hd), g)
    k, v = [[_normal((c + n, G, hd), g) for c, n in lens] for _ in range(2)]
    return lens, q, k, v


def _prepare_attention(case, seed):
    lens, q, k, v = _attention_inputs(case, seed)
    G, hd = case["kv_heads"], case["head_dim"]
    cache = SequenceCache([CacheSpec.kv(G, hd)], max_tokens=sum((c + n + 63) // 64 * 64 for c, n in lens), max_seqs=len(lens),
                          device=DEVICE, max_seq_tokens=max(c + n for c, n in lens))
    slots = [cache.allocate() for _ in lens]
    left = dict(zip(slots, [c for c, _ in lens]))
    while any(left.values()):                                    # sequences that grow side by side take pages in turn
        for slot in slots:
            n = min(left[slot], 64)
            if n:
                cache.reserve([(slot, n)])
                cache.advance(slot, n)
                left[slot] -= n
    cache.reserve([(slot, n) for slot, (_, n) in zip(slots, lens)])
    step = build_step_batch([(slot, [0] * n) for slot, (_, n) in zip(slots, lens)], [[]] * len(lens), cache, DEVICE)
    group = cache.kv_groups[0]
    for slot, ks, vs in zip(slots, k, v):
        for b, page in enumerate(group.pages[slot]):
            rows = slice(64 * b, 64 * b + 64)
            for pages, rows_of in ((group.k[0], ks), (group.v[0], vs)):
                part = rows_of[rows].transpose(0, 1)
                pages[page, :, :part.shape[1]] = part
    kv = KVLayerCache(group.k[0], group.v[0], step.block_tables[0], case["window"] or None, True)
    return dict(kind="attention", q=q, kv=kv, step=step, kv_heads=G, scale=hd ** -0.5)


def _run_attention(s):
    return ops.attention(s["q"], s["kv"], s["step"], s["kv_heads"], s["scale"])


def _exact_attention(case, seed):
    lens, q, k, v = _attention_inputs(case, seed)
    out, at = [], 0
    for (c, n), ks, vs in zip(lens, k, v):
        out.append(_attend(q[at:at + n].double(), ks.double(), vs.double(), c, case["head_dim"] ** -0.5, case["window"]))
        at += n
    return torch.cat(out)


# -------------------------------------------------------------------------------------- single layers: parts
def _part(case):
    rt = Runtime(torch.device(DEVICE), torch.bfloat16)
    if case["kind"] == "mlp":
        return build_part("feed_forward", PartSpec("gated_mlp", {
            "hidden_size": case["width"], "intermediate_size": case["ff"], "activation": "silu", "gate_name": "gate",
            "up_name": "up", "down_name": "down"}), rt)
    if case["kind"] == "routed":
        return build_part("feed_forward", PartSpec("routed_mlp", {
            "hidden_size": case["width"], "experts": case["experts"], "top": case["top"], "expert_size": case["ff"],
            "route_scale": 2.0, "activation": "silu" if case["gated"] else "relu2", "router_name": "router", "expert_prefix": "e",
            "gate_name": "gate", "up_name": "up", "down_name": "down",
            "groups": {"count": case["groups"], "keep": 2} if case["groups"] > 1 else None,
            "shared": {"size": case["shared"], "prefix": "shared"} if case["shared"] else None}), rt)
    if case["kind"] == "gla":
        return build_part("mixer", PartSpec("gla", {
            "hidden_size": case["width"], "heads": case["heads"], "dim": case["dim"], "vdim": case["vdim"], "tau": 16.0,
            "decay_rank": 16, "eps": EPS}), rt)
    if case["kind"] == "delta":
        more = {"decay": "head", "gate": "full", "gate_activation": "silu"} if case["decay"] == "head" else {"rank": 16}
        return build_part("mixer", PartSpec("gated_delta", {
            "hidden_size": case["width"], "heads": case["heads"], "kv_heads": case["kv_heads"], "dim": case["dim"], "vdim": case["vdim"],
            "conv": 4, "eps": EPS, **more}), rt)
    return build_part("mixer", PartSpec("retention", {
        "hidden_size": case["width"], "heads": case["heads"], "dim": case["dim"], "vdim": case["vdim"], "decay": _decays(case["heads"]),
        "eps": EPS, "position": PartSpec("rope", {"head_dim": case["dim"], "rotary_dim": case["dim"], "theta": ROPE_THETA,
                                                  "scaling": None, "pairing": "half", "max_positions": 1 << 30})}), rt)


def _decays(heads):
    return [1.0 - 2.0 ** (-5.0 - 6.0 * h / max(1, heads - 1)) for h in range(heads)]


def _part_inputs(case, seed, part):
    """A layer's tensors and its normed input rows."""
    g = _generator(seed)
    tensors = _tensors(part.weight_specs(), g)
    n = case["tokens"] if "seqs" not in case else sum(_lengths(case["seqs"], case["tokens"]))
    return tensors, _normal((n, case["width"]), g)


def _prepare_feed_forward(case, seed):
    part = _part(case)
    tensors, h = _part_inputs(case, seed, part)
    part.load(tensors)
    return dict(kind="feed_forward", part=part, h=h)


def _run_feed_forward(s):
    delta = s["part"].forward(s["h"], None)
    return delta.compute() if hasattr(delta, "compute") else delta


def _prepare_mixer(case, seed):
    part = _part(case)
    tensors, h = _part_inputs(case, seed, part)
    part.load(tensors)
    lens = _lengths(case["seqs"], case["tokens"])
    if hasattr(part, "prepare"):
        part.prepare(max(lens))
    cache = SequenceCache([part.cache_spec()], max_tokens=sum((n + 63) // 64 * 64 for n in lens), max_seqs=len(lens), device=DEVICE,
                          max_seq_tokens=max(lens))
    slots = [cache.allocate() for _ in lens]
    cache.reserve(list(zip(slots, lens)))
    step = build_step_batch([(slot, [0] * n) for slot, n in zip(slots, lens)], [[]] * len(lens), cache, DEVICE)
    return dict(kind="mixer", part=part, h=h, step=step, state=StateLayerCache(cache.state[0]))


def _run_mixer(s):
    """The layer's delta and the sequences' states, which every pass carries on."""
    delta = s["part"].forward(s["h"], s["step"], s["state"])
    return {"delta": delta.compute() if hasattr(delta, "compute") else delta, "state": s["state"].state}


def _exact_mlp(case, seed):
    w, h = _part_inputs(case, seed, _part(case))
    h = h.double()
    return (torch.nn.functional.silu(h @ w["gate"].double().T) * (h @ w["up"].double().T)) @ w["down"].double().T


def _exact_routed(case, seed):
    w, h = _part_inputs(case, seed, _part(case))
    h = h.double()
    E, top, T = case["experts"], case["top"], h.shape[0]
    scores = torch.sigmoid(h @ w["router"].double().T)
    choice = scores
    if case["groups"] > 1:
        per = choice.view(T, case["groups"], -1)
        kept = per.topk(2, -1).values.sum(-1).topk(2, -1).indices
        mask = torch.zeros((T, case["groups"]), dtype=torch.bool, device=DEVICE).scatter_(1, kept, True)
        choice = per.masked_fill(~mask[:, :, None], -1.0).reshape(T, E)
    ids = choice.topk(top, -1).indices
    weight = scores.gather(1, ids)
    weight = 2.0 * weight / weight.sum(-1, keepdim=True)
    out = torch.zeros((T, case["width"]), dtype=torch.float64, device=DEVICE)

    def expert(x, at):
        up = x @ w[at + "up"].double().T
        act = torch.nn.functional.silu(x @ w[at + "gate"].double().T) * up if case["gated"] else torch.relu(up) ** 2
        return act @ w[at + "down"].double().T

    for e in range(E):
        t, k = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            out.index_add_(0, t, weight[t, k][:, None] * expert(h[t], f"e{e}."))
    return out + expert(h, "shared.") if case["shared"] else out


def _group_norm(x, size):
    return (x.view(x.shape[0], -1, size) * torch.rsqrt((x.view(x.shape[0], -1, size) ** 2).mean(-1, keepdim=True) + EPS))


def _scan(q, k, v, decay, delta=None):
    """S <- decay S (per key channel); S <- S + k u^T with u = v, or beta (v - S^T k) for a delta rule; o = S^T q.  q, k, decay
    [T, H, N], v [T, H, P], delta [T, H]; returns (o [T, H, P], S)."""
    T, H, N = k.shape
    S = torch.zeros((H, N, v.shape[2]), dtype=torch.float64, device=v.device)
    out = torch.empty_like(v)
    for t in range(T):
        S = S * decay[t, :, :, None]
        u = v[t] if delta is None else delta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
        out[t] = torch.bmm(q[t, :, None], S)[:, 0]
    return out, S


def _exact_mixer(case, seed):
    w, h = _part_inputs(case, seed, _part(case))
    w = {name: t.double() for name, t in w.items()}
    H, N, P = case["heads"], case["dim"], case["vdim"]
    silu = torch.nn.functional.silu
    deltas, states, at = [], [], 0
    for n in _lengths(case["seqs"], case["tokens"]):
        x = h[at:at + n].double()
        at += n
        if case["kind"] == "gla":
            q, k = ((x @ w[name].T).view(n, H, N) for name in "qk")
            alpha = torch.sigmoid((x @ w["a1"].T) @ w["a2"].T + w["a2.b"]) ** (1.0 / 16.0)
            o, S = _scan(q * N ** -0.5, k, (x @ w["v"].T).view(n, H, P), alpha.view(n, H, N))
            o = _group_norm(o.reshape(n, -1), P) * w["norm"]
            o = o.reshape(n, -1) * silu(x @ w["g"].T)
        elif case["kind"] == "retention":
            angle = torch.arange(n, dtype=torch.float64, device=DEVICE)[:, None, None] * ROPE_THETA ** (
                -torch.arange(0, N, 2, dtype=torch.float64, device=DEVICE) / N)
            q, k = ((x @ w[name].T).view(n, H, N) for name in "qk")
            q, k = (torch.cat([a[..., :N // 2] * angle.cos() - a[..., N // 2:] * angle.sin(),
                               a[..., N // 2:] * angle.cos() + a[..., :N // 2] * angle.sin()], -1) for a in (q, k))
            decay = torch.tensor(_decays(H), dtype=torch.float64, device=DEVICE).view(1, H, 1).expand(n, H, N)
            o, S = _scan(q, k * N ** -0.5, (x @ w["v"].T).view(n, H, P), decay)
            o = _group_norm(o.reshape(n, -1), P).reshape(n, -1) * silu(x @ w["g"].T)
        else:
            G = case["kv_heads"]
            raw = torch.cat([x @ w[name].T for name in "qkv"], 1)
            taps = torch.cat([w[name + ".conv"] for name in "qkv"])
            back = torch.cat([torch.zeros((3, raw.shape[1]), dtype=torch.float64, device=DEVICE), raw])
            mixed = silu(sum(back[i:i + n] * taps[:, i] for i in range(4)))
            q, k = (mixed[:, i * G * N:(i + 1) * G * N].view(n, G, N) for i in (0, 1))
            q, k = (a * torch.rsqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
            q, k = (a.repeat_interleave(H // G, 1) for a in (q * N ** -0.5, k))
            channel = case["decay"] == "channel"
            z = (x @ w["a1"].T) @ w["a2"].T if channel else x @ w["a"].T
            step = torch.nn.functional.softplus(z + w["dt_bias"]).view(n, H, -1)
            decay = torch.exp(-torch.exp(w["A_log"])[:, None] * step).expand(n, H, N)
            o, S = _scan(q, k, mixed[:, 2 * G * N:].view(n, H, P), decay, torch.sigmoid(x @ w["b"].T))
            o = (_group_norm(o.reshape(n, -1), P) * w["norm"]).reshape(n, -1)
            o = o * (torch.sigmoid((x @ w["g1"].T) @ w["g2"].T) if channel else silu(x @ w["g"].T))
        deltas.append(o @ w["o"].T)
        states.append(torch.cat([S.reshape(-1), back[-3:].reshape(-1)]) if case["kind"] == "delta" else S.reshape(-1))
    return {"delta": torch.cat(deltas), "state": torch.stack(states + [torch.zeros_like(states[0])])}


# ---------------------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    if case["kind"] == "llama":
        return _prepare_llama(case, seed)
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    return _prepare_feed_forward(case, seed) if case["kind"] in ("mlp", "routed") else _prepare_mixer(case, seed)


def run(state):
    return {"llama": _run_llama, "attention": _run_attention, "feed_forward": _run_feed_forward, "mixer": _run_mixer}[state["kind"]](state)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("llama", "attention", "mlp", "routed"):
        return {"llama": _exact_llama, "attention": _exact_attention, "mlp": _exact_mlp, "routed": _exact_routed}[kind](case, seed)
    return _exact_mixer(case, seed)


def work(case):
    kind = case["kind"]
    item = 4 if case.get("dtype") == "float32" else 2
    if kind == "llama":
        d, ff, H, G, hd = (case[k] for k in ("width", "ff", "heads", "kv_heads", "head_dim"))
        layer = d * (2 * H + 2 * G) * hd + 3 * d * ff
        lens = _lengths(case["seqs"], case["prompt"])
        rows = sum(lens) if case["want"] == "all" else len(lens)
        head = d * case["vocab"]
        pairs = sum(n * (n + 1) // 2 for n in lens)
        kv = 2 * G * hd * item * case["layers"]
        flops = 2 * sum(lens) * layer * case["layers"] + 4 * pairs * H * hd * case["layers"] + 2 * rows * head
        total = (layer * case["layers"] + head) * item + sum(lens) * kv + rows * case["vocab"] * 4
        for i in range(case["new"]):
            keys = sum(n + i + 1 for n in lens)
            flops += 2 * len(lens) * (layer * case["layers"] + head) + 4 * keys * H * hd * case["layers"]
            total += (layer * case["layers"] + head) * item + keys * kv + len(lens) * case["vocab"] * 4
        return {"bytes": total, "flops": flops}
    if kind == "attention":
        H, G, hd, w = case["heads"], case["kv_heads"], case["head_dim"], case["window"]
        lens = _attention_lengths(case)
        pairs = sum(min(c + i + 1, w) if w else c + i + 1 for c, n in lens for i in range(n))
        keys = sum(min(c, w) + n if w else c + n for c, n in lens)
        return {"bytes": 2 * (2 * sum(n for _, n in lens) * H * hd + 2 * keys * G * hd), "flops": 4 * pairs * H * hd}
    d = case["width"]
    if kind in ("mlp", "routed"):
        T = case["tokens"]
        rows = 6 * T * d
        if kind == "mlp":
            return {"bytes": 2 * 3 * d * case["ff"] + rows, "flops": 2 * T * 3 * d * case["ff"]}
        E, per = case["experts"], (3 if case["gated"] else 2) * d * case["ff"]
        used = E * (1.0 - (1.0 - case["top"] / E) ** T)             # experts that some token chooses, for even choices
        shared = 3 * d * case["shared"]
        return {"bytes": 2 * (used * per + shared + E * d) + rows, "flops": 2 * T * (case["top"] * per + shared + E * d)}
    lens = _lengths(case["seqs"], case["tokens"])
    T, H, N, P = sum(lens), case["heads"], case["dim"], case["vdim"]
    G = case.get("kv_heads", H)
    weights = d * (2 * G * N + 3 * H * P)
    state = len(lens) * H * N * P * 4
    return {"bytes": 2 * weights + 6 * T * d + 2 * state, "flops": 2 * T * weights + (8 if kind == "delta" else 4) * T * H * N * P}


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 5e-6}
    return {"rel": 3e-2 if case["kind"] == "llama" else 1e-2}
