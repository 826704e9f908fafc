"""The work this framework is measured on: calls that a program which serves models makes, through the parts, the cache
manager and the step function, at the sizes of the repository's own benchmark and around them.

A case names a kind of layer (or a whole model), its sizes and the ragged batch it runs:

  serve     a whole Llama: the step function runs several prompts, then single tokens of all requests; logits come back
  block     one pre-norm block of grouped-query attention and SwiGLU (what a Llama is made of)
  experts   a routed feed-forward
  latent    attention over a low-rank latent
  scan      a state-space layer (Mamba-2)
  linear    linear attention with a decay per head
  window    attention over a sliding window plus averaged blocks

``tokens`` new tokens are shared out over ``requests`` requests, the first the longest; ``past`` tokens (fewer for the later
requests) are cached before.  With one token a request the layer's launches are captured in a CUDA graph once and
replayed, as the step function does with decode steps; anything longer is issued call by call, as it does with prompts.
Every layer's exact value is worked out here in 64 bits with plain torch.
"""
import math
import random

import torch

from torchinferno_b200.cache.manager import CacheManager
from torchinferno_b200.engine.batch import EntryPlacement, StepEntry, build_batch
from torchinferno_b200.engine.factory import make_runner, random_model
from torchinferno_b200.kernels import gemm, ops
from torchinferno_b200.parts.base import KVBinding, LayerContext, PartSpec, ResidualStream, build_part

DEVICE = "cuda"
PAGE = 16
EPS = 1e-6
THETA = 500000.0


def listed():
    return [
        # A small chat model (the 1B sizes) as a server runs it: eight prompts in one step, then four decode steps.
        {"name": "serve_1b", "kind": "serve", "layers": 16, "width": 2048, "heads": 32, "kv_heads": 8, "dim": 64, "ff": 8192,
         "vocab": 128256, "requests": 8, "tokens": 1900, "new": 4},
        # One layer of the 8B sizes on a prefill step: a long prompt, two shorter ones behind cached context.
        {"name": "block_prompt", "kind": "block", "dtype": "bf16", "width": 4096, "heads": 32, "kv_heads": 8, "dim": 128, "ff": 14336,
         "requests": 3, "tokens": 2048, "past": 512},
        # The same layer on the headline decode step: eight requests at up to 4,096 tokens.
        {"name": "block_decode", "kind": "block", "dtype": "bf16", "width": 4096, "heads": 32, "kv_heads": 8, "dim": 128, "ff": 14336,
         "requests": 8, "tokens": 8, "past": 4090},
        # The 32-bit path, for checking a checkpoint: one layer of the 1B sizes on two short prompts.
        {"name": "block_f32", "kind": "block", "dtype": "f32", "width": 2048, "heads": 32, "kv_heads": 8, "dim": 64, "ff": 8192,
         "requests": 2, "tokens": 301, "past": 0},
        # Routed experts on a prompt, with a gated shared expert.
        {"name": "experts_prompt", "kind": "experts", "width": 2048, "ff": 1024, "experts": 32, "top": 4, "shared": 2048,
         "activation": "relu2", "tokens": 2048},
        # Clamped gated experts on a decode step of eight requests: the chosen experts' weights are the work.
        {"name": "experts_decode", "kind": "experts", "width": 2048, "ff": 1024, "experts": 32, "top": 4, "shared": 2048,
         "activation": "glu_clamp", "tokens": 8},
        # Latent attention on a long prompt beside a short one.
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "heads": 16, "dim": 128, "rank": 512, "rot": 64, "q_rank": 0,
         "gate": "element", "sink": False, "requests": 2, "tokens": 2500, "past": 0},
        # The same on a decode step, queries through a latent of their own.
        {"name": "latent_decode", "kind": "latent", "width": 2048, "heads": 16, "dim": 128, "rank": 512, "rot": 64, "q_rank": 768,
         "gate": "head", "sink": False, "requests": 8, "tokens": 8, "past": 3000},
        # A state-space layer on two prompts.
        {"name": "scan_prompt", "kind": "scan", "width": 2048, "heads": 64, "dim": 64, "state": 128, "groups": 1, "norm_groups": 1,
         "requests": 2, "tokens": 2048},
        # Linear attention on two prompts, and on a decode step (the smallest call).
        {"name": "linear_prompt", "kind": "linear", "width": 2048, "heads": 16, "dim": 128, "requests": 2, "tokens": 2048},
        {"name": "linear_decode", "kind": "linear", "width": 2048, "heads": 16, "dim": 128, "requests": 8, "tokens": 8},
        # Attention in a window of 512 with blocks of 64, a prompt behind cached context.
        {"name": "window_prompt", "kind": "window", "width": 2048, "heads": 16, "kv_heads": 8, "dim": 128, "window": 512, "pool": 64,
         "extras": True, "requests": 2, "tokens": 2048, "past": 700},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["block", "block", "experts", "experts", "latent", "latent", "scan", "linear", "window"])
    requests = _spread(rng, 1, 12)
    single = rng.random() < 0.4                       # a decode step
    tokens = requests if single else max(requests + 1, _spread(rng, 20, 2600))
    past = _spread(rng, 1, 4000) if single else rng.choice([0, _spread(rng, 1, 1500)])
    if not single:
        requests = min(requests, 4, tokens - 1)
    heads = rng.choice([4, 8, 12, 16, 24, 32])
    width = 64 * rng.randint(8, 48)
    if kind == "block":
        f32 = rng.random() < 0.2
        if f32:
            tokens, past = (tokens, min(past, 300)) if single else (max(requests + 1, min(tokens, 300)), min(past, 100))
        return {"kind": "block", "dtype": "f32" if f32 else "bf16", "width": min(width, 1536) if f32 else width, "heads": heads,
                "kv_heads": heads // rng.choice([1, 2, 4]), "dim": rng.choice([64, 128]), "ff": 32 * rng.randint(16, 100 if f32 else 300),
                "requests": requests, "tokens": tokens, "past": past}
    if kind == "experts":
        experts = rng.choice([8, 16, 28, 32, 60])
        return {"kind": "experts", "width": min(width, 2560), "ff": 32 * rng.randint(8, 48), "experts": experts, "top": rng.randint(1, 6),
                "shared": rng.choice([0, 512, 2048]), "activation": rng.choice(["relu2", "gelu", "swiglu", "glu_clamp"]),
                "tokens": tokens}
    if kind == "latent":
        return {"kind": "latent", "width": width, "heads": heads, "dim": rng.choice([64, 128]), "rank": rng.choice([128, 256, 512, 512]),
                "rot": rng.choice([32, 64]), "q_rank": rng.choice([0, 768]), "gate": rng.choice(["element", "head"]),
                "sink": rng.random() < 0.4, "requests": requests, "tokens": tokens, "past": past}
    if kind == "scan":
        return {"kind": "scan", "width": width, "heads": 4 * rng.randint(4, 20), "dim": rng.choice([32, 64, 64, 128]),
                "state": rng.choice([64, 128, 128]), "groups": rng.choice([1, 1, 2, 4]), "norm_groups": rng.choice([1, 4]),
                "requests": requests, "tokens": tokens}
    if kind == "linear":
        return {"kind": "linear", "width": width, "heads": heads, "dim": rng.choice([64, 128, 128]), "requests": requests, "tokens": tokens}
    return {"kind": "window", "width": width, "heads": heads, "kv_heads": heads // rng.choice([1, 2, 4]), "dim": rng.choice([64, 128]),
            "window": _spread(rng, 64, 1024), "pool": rng.choice([0, 16, 64]), "extras": rng.random() < 0.5,
            "requests": requests, "tokens": tokens, "past": past}


# ------------------------------------------------------------------------------------------------ batch and random values
def portions(case):
    """(new tokens, cached tokens) of every request."""
    n, total = case["requests"], case["tokens"]
    share = [1.0 / (i + 1) for i in range(n)]
    lens = [max(1, int(total * s / sum(share))) for s in share]
    lens[0] += total - sum(lens)
    past = case.get("past", 0)
    return lens, [max(0, past - i * (past // (2 * n))) for i in range(n)]


class Values:
    """Random tensors from a seed, in one order."""

    def __init__(self, seed, dtype):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed) * 1000003 + 17)
        self.dtype = dtype

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        t = torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(mean, std, generator=self.g)
        return t.to(self.dtype if dtype is None else dtype)

    def matrix(self, rows, cols, std=None):
        return self.normal(rows, cols, std=cols ** -0.5 if std is None else std)

    def vector(self, n, std=1.0, mean=0.0):
        return self.normal(n, std=std, mean=mean, dtype=torch.bfloat16).float()


def dtype_of(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


def inputs(case, seed):
    """(weights by name, rows the layer reads, what is cached or carried before the step), all from the seed."""
    v, kind, w = Values(seed, dtype_of(case)), case["kind"], case["width"]
    n, (lens, pasts) = case["tokens"], portions(case) if "requests" in case else ([], [])
    held = sum(pasts)
    if kind == "block":
        h, k, d, ff = case["heads"], case["kv_heads"], case["dim"], case["ff"]
        weights = {"norm1.weight": v.vector(w, 0.1, 1.0), "a.q_proj.weight": v.matrix(h * d, w), "a.k_proj.weight": v.matrix(k * d, w),
                   "a.v_proj.weight": v.matrix(k * d, w), "a.o_proj.weight": v.matrix(w, h * d), "norm2.weight": v.vector(w, 0.1, 1.0),
                   "m.gate_proj.weight": v.matrix(ff, w), "m.up_proj.weight": v.matrix(ff, w), "m.down_proj.weight": v.matrix(w, ff)}
        return weights, v.normal(n, w, dtype=torch.float32), {"k": v.normal(held, k, d), "v": v.normal(held, k, d)}
    if kind == "experts":
        e, ff, s, act = case["experts"], case["ff"], case["shared"], case["activation"]
        weights = {"router": v.matrix(e, w, 2 * w ** -0.5)}
        gated = act in ("glu_clamp", "swiglu")
        for prefix, size in [(f"e{i}.", ff) for i in range(e)] + ([("shared.", s)] if _shared(case) else []):
            if gated:
                weights[prefix + "gate"] = v.matrix(size, w)
            weights[prefix + "up"], weights[prefix + "down"] = v.matrix(size, w), v.matrix(w, size)
        if _shared(case):
            weights["shared.sg"] = v.matrix(1, w)
        return weights, v.normal(n, w), {}
    if kind == "latent":
        h, d, c, r, qr = case["heads"], case["dim"], case["rank"], case["rot"], case["q_rank"]
        weights = {"q": v.matrix(h * (d + r), w)} if not qr else {
            "dq": v.matrix(qr, w), "dq.norm": v.vector(qr, 0.1, 1.0), "uq": v.matrix(h * (d + r), qr)}
        weights.update({"dkv": v.matrix(c + r, w), "dkv.norm": v.vector(c, 0.1, 1.0), "uk": v.matrix(h * d, c), "uv": v.matrix(h * d, c),
                        "g": v.matrix(h if case["gate"] == "head" else h * d, w), "o": v.matrix(w, h * d)})
        if case["sink"]:
            weights["sink"] = v.vector(h)
        return weights, v.normal(n, w), {"latent": v.normal(held, c + r)}
    if kind == "scan":
        h, p, s, g = case["heads"], case["dim"], case["state"], case["groups"]
        inner, channels = h * p, h * p + 2 * g * s
        weights = {"in": v.matrix(inner + channels + h, w), "conv": v.normal(channels, 4, std=0.5, dtype=torch.bfloat16).float(),
                   "conv.b": v.vector(channels, 0.1), "dt_bias": v.vector(h), "A_log": v.vector(h, 0.5), "D": v.vector(h, 0.3, 1.0),
                   "norm": v.vector(inner, 0.1, 1.0), "o": v.matrix(w, inner)}
        carried = [v.normal(h * s * p, std=0.5, dtype=torch.float32) for _ in lens]
        before = [v.normal(3 * channels, dtype=torch.bfloat16).float() for _ in lens]
        return weights, v.normal(n, w), {"state": torch.stack([torch.cat(pair) for pair in zip(carried, before)])}
    if kind == "linear":
        h, d = case["heads"], case["dim"]
        weights = {name: v.matrix(h * d, w) for name in ("q", "k", "v", "g")}
        weights.update({"o": v.matrix(w, h * d), "norm": v.vector(h * d, 0.1, 1.0)})
        return weights, v.normal(n, w), {"state": v.normal(len(lens), h, d, d, std=0.5, dtype=torch.float32)}
    h, k, d = case["heads"], case["kv_heads"], case["dim"]
    weights = {"q": v.matrix(h * d, w), "k": v.matrix(k * d, w), "v": v.matrix(k * d, w), "o": v.matrix(w, h * d)}
    if case["extras"]:
        weights.update({"q.b": v.vector(h * d, 0.5), "k.b": v.vector(k * d, 0.5), "v.b": v.vector(k * d, 0.5), "temp": v.vector(h, 0.2, 1.0),
                        "sink": v.vector(h), "g": v.matrix(h * d, w)})
    blocks = sum(past // case["pool"] for past in pasts) if case["pool"] else 0
    return weights, v.normal(n, w), {"k": v.normal(held, k, d), "v": v.normal(held, k, d), "mean_k": v.normal(blocks, k, d, std=0.2),
                                     "mean_v": v.normal(blocks, k, d, std=0.2)}


def _shared(case):
    return case["shared"] if case["activation"] != "swiglu" else 0      # (a plain gated unit has no shared form)


# ----------------------------------------------------------------------------------------------------- the framework's side
def part_of(case):
    """The layer, by category and description."""
    kind, w = case["kind"], case["width"]
    if kind == "block":
        position = PartSpec("rotary", {"head_dim": case["dim"], "theta": THETA, "exact": True})
        mixer = PartSpec("gqa_attention", {"hidden_size": w, "heads": case["heads"], "kv_heads": case["kv_heads"], "head_dim": case["dim"],
                                           "position": position}, prefix="a.")
        norm = {"width": w, "eps": EPS}
        return "block", PartSpec("prenorm", {
            "mixer": mixer, "feed_forward": PartSpec("swiglu", {"hidden_size": w, "intermediate_size": case["ff"]}, prefix="m."),
            "mixer_norm": PartSpec("rmsnorm", norm, prefix="norm1."), "feed_forward_norm": PartSpec("rmsnorm", norm, prefix="norm2.")})
    if kind == "experts":
        act = case["activation"]
        return "feed_forward", PartSpec("routed_experts", {
            "hidden_size": w, "experts": case["experts"], "top": case["top"], "expert_size": case["ff"], "activation": act,
            "scores": "sigmoid" if act == "glu_clamp" else "softmax", "normalize": act != "glu_clamp", "norm_eps": 0.0 if act == "glu_clamp" else 1e-20,
            "shared_size": _shared(case), "shared_gate": bool(_shared(case)), "limit": 7.0 if act == "glu_clamp" else 0.0,
            "weight_on_input": act == "glu_clamp"})
    if kind == "latent":
        return "mixer", PartSpec("latent_attention", {
            "hidden_size": w, "heads": case["heads"], "dim": case["dim"], "rot_dim": case["rot"], "value_dim": case["dim"],
            "kv_rank": case["rank"], "scale": (case["dim"] + case["rot"]) ** -0.5, "rot_base": THETA, "eps": EPS, "gate": case["gate"],
            "sink": case["sink"], "q_rank": case["q_rank"], "pairing": "half" if case["q_rank"] else "interleaved"})
    if kind == "scan":
        return "mixer", PartSpec("state_space_duality", {
            "hidden_size": w, "heads": case["heads"], "head_dim": case["dim"], "state_dim": case["state"], "groups": case["groups"],
            "norm_groups": case["norm_groups"], "eps": EPS})
    if kind == "linear":
        return "mixer", PartSpec("decay_linear_attention", {
            "hidden_size": w, "heads": case["heads"], "key_dim": case["dim"], "value_dim": case["dim"], "decay": decays(case["heads"]), "eps": EPS})
    x = case["extras"]
    return "mixer", PartSpec("pooled_window_attention", {
        "hidden_size": w, "heads": case["heads"], "kv_heads": case["kv_heads"], "dim": case["dim"], "value_dim": case["dim"],
        "scale": case["dim"] ** -0.5, "position": PartSpec("rotary", {"head_dim": case["dim"], "theta": THETA, "rot_dim": 64, "exact": True}),
        "window": case["window"], "pool": case["pool"] or None, "value_rotation_base": THETA if x else None, "bias": x, "sink": x,
        "temperature": x, "gate": x})


def decays(heads):
    return [1 - 2.0 ** -(3 + i % 6) for i in range(heads)]


class Prepared:
    """A bound layer with its cache and one step's batch, or a model with its runner."""
    graph = None
    outputs = None


def prepare(case, seed):
    if case["kind"] == "serve":
        return _prepare_serve(case, seed)
    s, dtype = Prepared(), dtype_of(case)
    weights, s.x, before = inputs(case, seed)
    category, spec = part_of(case)
    s.part = build_part(category, spec, dtype=dtype, device=torch.device(DEVICE))
    if category == "block":
        for prefix, part in s.part.named_parts():
            part.bind({ws.name: weights[prefix + ws.name] for ws in part.weight_specs()})
    else:
        s.part.bind(weights)
    gemm.tune_few_rows()      # (what a model does once all its weights are bound)
    s.category, s.ctx, s.initial = category, LayerContext(batch=None), None
    if case["kind"] != "experts":
        _fill_cache(case, s, before, dtype)
    if case["tokens"] == case.get("requests", case["tokens"] if case["tokens"] <= 16 else 0):
        _pass(s)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            s.outputs = _pass(s)
        torch.cuda.synchronize()
    return s


def _fill_cache(case, s, before, dtype):
    mixer = s.part.mixer if s.category == "block" else s.part
    specs = [spec for spec in (mixer.cache_spec(), mixer.side_cache_spec()) if spec is not None]
    lens, pasts = portions(case)
    longest = max(a + b for a, b in zip(lens, pasts))
    cache = CacheManager(specs, [mixer.state_spec()], page_size=PAGE, num_pages=sum(-(-(a + b) // PAGE) + 1 for a, b in zip(lens, pasts)),
                         max_requests=len(lens), max_request_tokens=longest, dtype=dtype, device=DEVICE)
    for group in cache.groups:
        if group.pool is not None:
            group.pool.zero_()
    placements, row = [], 0
    for i, (new, past) in enumerate(zip(lens, pasts)):
        cache.open(i)
        if past:
            cache.extend(i, past)
        cache.extend(i, new)
        placements.append(EntryPlacement(i, cache.slot(i), row, new, past))
        row += new
    batch, updates = build_batch(placements, [[0] * n for n in lens], [[n - 1] for n in lens],
                                 cache.drain_table_updates() + [cache.drain_record_updates()], cache.device)
    for target, (index, value) in zip([group.table_device for group in cache.groups] + [cache.request_records], updates):
        if index.numel():
            ops.scatter_i32(target, index, value)
    bindings = []
    for layer in range(len(specs)):
        b = cache.kv_binding(layer)
        bindings.append(KVBinding(b.pool, b.block_table, b.page_size, b.window, True, b.keys, b.values))
    s.cache = cache
    s.ctx = LayerContext(batch=batch, kv=bindings[0] if bindings else None, side_kv=bindings[1] if len(bindings) > 1 else None,
                         state=cache.state(0), error_word=cache.error_word)
    gemm.set_error_word(cache.error_word)
    if "state" in before:
        s.initial = torch.empty_like(s.ctx.state)
        for i in range(len(lens)):
            s.initial[cache.slot(i)] = before["state"][i].view(s.initial.shape[1:])
    held = {"latent": (0, "keys"), "k": (0, "keys"), "v": (0, "values"), "mean_k": (1, "keys"), "mean_v": (1, "values")}
    for name, rows in before.items():
        if name not in held or not rows.numel():
            continue
        layer, which = held[name]
        pages, first = getattr(bindings[layer], which), 0
        for i, past in enumerate(pasts):
            count = past // case["pool"] if layer else past
            at = torch.arange(count, device=DEVICE)
            table = torch.tensor(cache.block_table(i, cache.group_of_layer(layer)), device=DEVICE)
            if count:
                source = rows[first:first + count]
                pages[table[at // PAGE], :, at % PAGE] = source.view(count, pages.shape[1], pages.shape[3])
            first += count


def _prepare_serve(case, seed):
    s = Prepared()
    config = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": case["vocab"], "hidden_size": case["width"],
              "intermediate_size": case["ff"], "num_hidden_layers": case["layers"], "num_attention_heads": case["heads"],
              "num_key_value_heads": case["kv_heads"], "head_dim": case["dim"], "max_position_embeddings": 8192, "rope_theta": THETA,
              "rope_scaling": None, "rms_norm_eps": 1e-5, "tie_word_embeddings": True}
    lens, _ = portions(case)
    model = random_model(config, seed, dtype="bfloat16")
    s.runner = make_runner(model, page_size=PAGE, max_tokens=case["tokens"] + case["requests"] * (case["new"] + PAGE),
                           max_requests=case["requests"], max_request_tokens=max(lens) + case["new"])
    rng = random.Random(seed)
    s.prompts = [[rng.randrange(case["vocab"]) for _ in range(n)] for n in lens]
    s.next = [[rng.randrange(case["vocab"]) for _ in lens] for _ in range(case["new"])]
    s.category = "serve"
    return s


def _pass(s):
    if s.category == "block":
        stream = ResidualStream(s.x.clone(), s.part.dtype)        # (a block adds to the residual in place)
        s.part.forward(stream, s.ctx)
        return {"residual": stream.settle(), "cache": s.ctx.kv.pool}
    if s.initial is not None:
        s.ctx.state.copy_(s.initial)                              # (the requests' state as the step finds it)
    y = s.part.forward(s.x, s.ctx)
    out = {"y": y}
    if s.initial is not None:
        out["state"] = s.ctx.state
    if s.ctx.kv is not None:
        out["cache"] = s.ctx.kv.pool
    return out


def run(s):
    if s.category == "serve":
        ids = list(range(len(s.prompts)))
        logits = [s.runner.step([StepEntry(i, p, [len(p) - 1]) for i, p in zip(ids, s.prompts)])]
        for tokens in s.next:
            logits.append(s.runner.step([StepEntry(i, [t], [0]) for i, t in zip(ids, tokens)]).clone())
        s.runner.end(ids)
        return logits
    if s.graph is not None:
        s.graph.replay()
        return s.outputs
    return _pass(s)


# ------------------------------------------------------------------------------------------------------------ work, tolerance
def work(case):
    kind, w, n = case["kind"], case["width"], case["tokens"]
    size = 4 if case.get("dtype") == "f32" else 2
    if kind == "serve":
        lens, _ = portions(case)
        layer = w * case["heads"] * case["dim"] * 2 + 2 * w * case["kv_heads"] * case["dim"] + 3 * w * case["ff"]
        head, r, new = w * case["vocab"], case["requests"], case["new"]
        kv = 2 * case["kv_heads"] * case["dim"] * 2 * case["layers"]
        return {"bytes": (1 + new) * (case["layers"] * layer + head) * 2 + kv * n * (1 + new) + 4 * case["vocab"] * r * (1 + new),
                "flops": 2 * case["layers"] * layer * (n + r * new) + 2 * head * r * (1 + new)
                + case["layers"] * 4 * case["heads"] * case["dim"] * (sum(m * m / 2 for m in lens) + n * new)}
    if kind == "experts":
        e, top, ff, s = case["experts"], case["top"], case["ff"], _shared(case)
        mats = 3 if case["activation"] in ("glu_clamp", "swiglu") else 2
        touched = e * (1 - (1 - top / e) ** n)
        return {"bytes": 2 * mats * w * (touched * ff + s) + 4 * e * w + 4 * n * w, "flops": 2 * n * w * (mats * (top * ff + s) + e)}
    lens, pasts = portions(case)
    pairs = sum(m * p + m * (m + 1) / 2 for m, p in zip(lens, pasts))          # (query, key) pairs of causal attention
    keys = sum(m + p for m, p in zip(lens, pasts))
    if kind == "block":
        h, k, d, ff = case["heads"], case["kv_heads"], case["dim"], case["ff"]
        mats = 2 * w * h * d + 2 * w * k * d + 3 * w * ff
        return {"bytes": size * (mats + 2 * k * d * (keys + n)) + 8 * n * w, "flops": 2 * n * mats + 4 * h * d * pairs}
    if kind == "latent":
        h, d, c, r = case["heads"], case["dim"], case["rank"], case["rot"]
        q = (w * case["q_rank"] + case["q_rank"] * h * (d + r)) if case["q_rank"] else w * h * (d + r)
        gate = w * (h if case["gate"] == "head" else h * d)
        mats = q + w * (c + r) + gate + w * h * d
        # (a prompt may make every head's keys and values from the latent; a single token is cheaper folded)
        unfolded = 2 * 2 * h * d * c * keys + 2 * h * (2 * d + r) * pairs
        folded = 2 * 2 * h * d * c * n + 2 * h * (2 * c + r) * pairs
        return {"bytes": 2 * (mats + 2 * h * d * c + (c + r) * (keys + n) + 2 * n * w), "flops": 2 * n * mats + min(unfolded, folded)}
    if kind == "scan":
        h, p, s, g = case["heads"], case["dim"], case["state"], case["groups"]
        inner = h * p
        mats = w * (2 * inner + 2 * g * s + h) + w * inner
        return {"bytes": 2 * mats + 4 * n * w + 8 * len(lens) * (h * s * p + 3 * (inner + 2 * g * s)), "flops": 2 * n * mats + 5 * n * inner * s}
    if kind == "linear":
        h, d = case["heads"], case["dim"]
        return {"bytes": 2 * 5 * w * h * d + 4 * n * w + 8 * len(lens) * h * d * d, "flops": 2 * n * 5 * w * h * d + 5 * n * h * d * d}
    h, k, d, win = case["heads"], case["kv_heads"], case["dim"], case["window"]
    mats = 2 * w * h * d + 2 * w * k * d + (w * h * d if case["extras"] else 0)
    seen = sum(min(p + t + 1, win) + ((p + t + 1 - win) // case["pool"] if case["pool"] and p + t + 1 > win else 0)
               for m, p in zip(lens, pasts) for t in range(m))
    read = sum(m + min(p, win) for m, p in zip(lens, pasts))
    return {"bytes": 2 * (mats + 2 * k * d * (read + n) + 2 * n * w), "flops": 2 * n * mats + 4 * h * d * seen}


def tolerance(case):
    if case.get("dtype") == "f32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "serve":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 1e-2, "max": 0.2}


# --------------------------------------------------------------------------------------------------- the exact values, 64 bits
def _rms(x, weight, eps=EPS):
    return x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt() * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, dims, pairing="half"):
    """Rotary positions over the first ``dims`` elements of the last dimension; x: [tokens, heads, width]."""
    freq = THETA ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)
    angle = pos.double()[:, None, None] * freq
    c, s, out = angle.cos(), angle.sin(), x.clone()
    lo, hi = (x[..., :dims // 2], x[..., dims // 2:dims]) if pairing == "half" else (x[..., 0:dims:2], x[..., 1:dims:2])
    a, b = lo * c - hi * s, hi * c + lo * s
    if pairing == "half":
        out[..., :dims // 2], out[..., dims // 2:dims] = a, b
    else:
        out[..., 0:dims:2], out[..., 1:dims:2] = a, b
    return out


def exact(case, seed):
    if case["kind"] == "serve":
        return None
    weights, x, before = inputs(case, seed)
    w = {name: t.double() for name, t in weights.items()}
    held = {name: t.double() for name, t in before.items()}
    return _EXACT[case["kind"]](case, w, x.double(), held)


def _requests(case):
    """(rows, past, cached rows) of every request, as slices."""
    row = first = 0
    for new, past in zip(*portions(case)):
        yield slice(row, row + new), past, slice(first, first + past)
        row, first = row + new, first + past


def _exact_block(case, w, x, held):
    h, k, d = case["heads"], case["kv_heads"], case["dim"]
    y = _rms(x, w["norm1.weight"])
    q, key, val = ((y @ w[f"a.{n}_proj.weight"].t()).view(len(x), -1, d) for n in "qkv")
    out = torch.empty(len(x), h * d, dtype=torch.float64, device=DEVICE)
    for rows, past, cached in _requests(case):
        pos = past + torch.arange(rows.stop - rows.start, device=DEVICE)
        qq = _rotate(q[rows], pos, d)
        kk = torch.cat([held["k"][cached], _rotate(key[rows], pos, d)]).repeat_interleave(h // k, 1)
        vv = torch.cat([held["v"][cached], val[rows]]).repeat_interleave(h // k, 1)
        score = torch.einsum("thd,shd->hts", qq, kk) * d ** -0.5
        score.masked_fill_(torch.arange(len(kk), device=DEVICE)[None, :] > pos[:, None], -math.inf)
        out[rows] = torch.einsum("hts,shd->thd", score.softmax(-1), vv).reshape(-1, h * d)
    x = x + out @ w["a.o_proj.weight"].t()
    y = _rms(x, w["norm2.weight"])
    x = x + (_silu(y @ w["m.gate_proj.weight"].t()) * (y @ w["m.up_proj.weight"].t())) @ w["m.down_proj.weight"].t()
    return {"residual": x, "cache": None}


def _exact_experts(case, w, x, held):
    act, top, e = case["activation"], case["top"], case["experts"]
    z = x @ w["router"].t()
    score = torch.sigmoid(z) if act == "glu_clamp" else z.softmax(-1)
    weight, ids = score.topk(top, -1)
    if act != "glu_clamp":
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)

    def expert(prefix, rows, scale=1.0):
        up = rows @ w[prefix + "up"].t() * scale
        if act == "relu2":
            inner = up.clamp(min=0) ** 2
        elif act == "gelu":
            inner = 0.5 * up * (1 + torch.erf(up * 0.5 ** 0.5))
        else:
            gate = rows @ w[prefix + "gate"].t() * scale
            if act == "swiglu":
                inner = _silu(gate) * up
            else:
                gate = gate.clamp(max=7.0)
                inner = gate * torch.sigmoid(1.702 * gate) * (up.clamp(-7.0, 7.0) + 1)
        return inner @ w[prefix + "down"].t()

    out = torch.zeros_like(x)
    for i in range(e):
        t, k = (ids == i).nonzero(as_tuple=True)
        if len(t):
            ww = weight[t, k][:, None]
            out.index_add_(0, t, expert(f"e{i}.", x[t], ww) if act == "glu_clamp" else ww * expert(f"e{i}.", x[t]))
    if _shared(case):
        out += torch.sigmoid(x @ w["shared.sg"].t()) * expert("shared.", x)
    return {"y": out}


def _exact_latent(case, w, x, held):
    h, d, c, r = case["heads"], case["dim"], case["rank"], case["rot"]
    pairing = "half" if case["q_rank"] else "interleaved"
    q = _rms(x @ w["dq"].t(), w["dq.norm"]) @ w["uq"].t() if case["q_rank"] else x @ w["q"].t()
    q, kv = q.view(len(x), h, d + r), x @ w["dkv"].t()
    latent, shared = _rms(kv[:, :c], w["dkv.norm"]), kv[:, c:]
    out = torch.empty(len(x), h, d, dtype=torch.float64, device=DEVICE)
    uk, uv = w["uk"].view(h, d, c), w["uv"].view(h, d, c)
    for rows, past, cached in _requests(case):
        pos = past + torch.arange(rows.stop - rows.start, device=DEVICE)
        qr = _rotate(q[rows][..., d:], pos, r, pairing)
        new = torch.cat([latent[rows], _rotate(shared[rows][:, None], pos, r, pairing)[:, 0]], 1)
        all_ = torch.cat([held["latent"][cached], new])
        folded = torch.cat([torch.einsum("thd,hdc->thc", q[rows][..., :d], uk), qr], -1)
        score = torch.einsum("thc,sc->hts", folded, all_) * (d + r) ** -0.5
        score.masked_fill_(torch.arange(len(all_), device=DEVICE)[None, :] > pos[:, None], -math.inf)
        if case["sink"]:
            score = torch.cat([score, w["sink"][:, None, None].expand(h, len(pos), 1)], -1)
        p = score.softmax(-1)[..., :len(all_)]
        out[rows] = torch.einsum("thc,hdc->thd", torch.einsum("hts,sc->thc", p, all_[:, :c]), uv)
    gate = torch.sigmoid(x @ w["g"].t())
    out = out * (gate[..., None] if case["gate"] == "head" else gate.view(len(x), h, d))
    return {"y": out.reshape(len(x), h * d) @ w["o"].t(), "cache": None}


def _exact_scan(case, w, x, held):
    h, p, s, g = case["heads"], case["dim"], case["state"], case["groups"]
    inner, channels, parts = h * p, h * p + 2 * g * s, case["norm_groups"]
    proj = x @ w["in"].t()
    z, u, dt = proj[:, :inner], proj[:, inner:inner + channels], proj[:, inner + channels:inner + channels + h]
    step = torch.nn.functional.softplus(dt + w["dt_bias"], threshold=1e9)
    decay = (-w["A_log"].exp() * step).exp()
    y, states = torch.empty(len(x), inner, dtype=torch.float64, device=DEVICE), []
    for i, (rows, _, _) in enumerate(_requests(case)):
        S, carried = held["state"][i][:h * s * p].view(h, s, p).clone(), held["state"][i][h * s * p:].view(3, channels)
        raw = torch.cat([carried, u[rows]])
        conv = _silu(sum(raw[j:j + rows.stop - rows.start] * w["conv"][:, j] for j in range(4)) + w["conv.b"])
        xs, B, C = conv[:, :inner].view(-1, h, p), conv[:, inner:inner + g * s].view(-1, g, s), conv[:, inner + g * s:].view(-1, g, s)
        B, C = B.repeat_interleave(h // g, 1), C.repeat_interleave(h // g, 1)
        dx = step[rows][..., None] * xs
        for t in range(len(xs)):
            S = decay[rows.start + t][:, None, None] * S + B[t][:, :, None] * dx[t][:, None, :]
            y[rows.start + t] = (torch.einsum("hsp,hs->hp", S, C[t]) + w["D"][:, None] * xs[t]).reshape(-1)
        states.append(torch.cat([S.reshape(-1), raw[-3:].reshape(-1)]))
    v = (y * _silu(z)).view(len(x), parts, inner // parts)
    v = v / (v.pow(2).mean(-1, keepdim=True) + EPS).sqrt()
    return {"y": (v.reshape(len(x), inner) * w["norm"]) @ w["o"].t(), "state": torch.stack(states)}


def _exact_linear(case, w, x, held):
    h, d = case["heads"], case["dim"]
    q, k, v = (_silu(x @ w[n].t()).view(len(x), h, d) for n in "qkv")
    lam = torch.tensor(decays(h), dtype=torch.float64, device=DEVICE)[:, None, None]
    y, states = torch.empty(len(x), h, d, dtype=torch.float64, device=DEVICE), []
    for i, (rows, _, _) in enumerate(_requests(case)):
        S = held["state"][i].clone()
        for t in range(rows.start, rows.stop):
            S = lam * S + k[t][:, :, None] * v[t][:, None, :]
            y[t] = torch.einsum("hkv,hk->hv", S, q[t])
        states.append(S)
    y = _rms(y.reshape(len(x), h * d), w["norm"]) * torch.sigmoid(x @ w["g"].t())
    return {"y": y @ w["o"].t(), "state": torch.stack(states)}


def _exact_window(case, w, x, held):
    h, k, d, win, pool, extras = case["heads"], case["kv_heads"], case["dim"], case["window"], case["pool"], case["extras"]
    q, key, val = ((x @ w[n].t() + (w[n + ".b"] if extras else 0.0)).view(len(x), -1, d) for n in "qkv")
    out = torch.empty(len(x), h, d, dtype=torch.float64, device=DEVICE)
    first_block = 0
    for rows, past, cached in _requests(case):
        n = rows.stop - rows.start
        pos, total = past + torch.arange(n, device=DEVICE), past + n
        qq, kk, vv = _rotate(q[rows], pos, 64), _rotate(key[rows], pos, 64), val[rows]
        if extras:
            qq = qq * w["temp"][:, None]
            vv = _rotate(vv, pos, d)
        kk, vv = torch.cat([held["k"][cached], kk]), torch.cat([held["v"][cached], vv])
        at = torch.arange(total, device=DEVICE)
        seen = (at[None] <= pos[:, None]) & (at[None] > pos[:, None] - win)
        if pool:
            old, count = past // pool, total // pool
            mean_k = torch.cat([held["mean_k"][first_block:first_block + old], kk[old * pool:count * pool].view(-1, pool, k, d).mean(1)])
            mean_v = torch.cat([held["mean_v"][first_block:first_block + old], vv[old * pool:count * pool].view(-1, pool, k, d).mean(1)])
            first_block += old
            end = (torch.arange(count, device=DEVICE) + 1) * pool - 1
            seen = torch.cat([seen, end[None] <= pos[:, None] - win], 1)
            kk, vv = torch.cat([kk, mean_k]), torch.cat([vv, mean_v])
        score = torch.einsum("thd,shd->hts", qq, kk.repeat_interleave(h // k, 1)) * d ** -0.5
        score.masked_fill_(~seen, -math.inf)
        if extras:
            score = torch.cat([score, w["sink"][:, None, None].expand(h, n, 1)], -1)
        o = torch.einsum("hts,shd->thd", score.softmax(-1)[..., :len(kk)], vv.repeat_interleave(h // k, 1))
        out[rows] = _rotate(o, -pos, d) if extras else o
    out = out.reshape(len(x), h * d)
    if extras:
        out = out * torch.sigmoid(x @ w["g"].t())
    return {"y": out @ w["o"].t(), "cache": None}


_EXACT = {"block": _exact_block, "experts": _exact_experts, "latent": _exact_latent, "scan": _exact_scan, "linear": _exact_linear,
          "window": _exact_window}
