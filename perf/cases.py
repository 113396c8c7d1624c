"""Cases that say how fast the framework is: the work that a program has it do, through the entry
points that it calls - a step of a whole model (``StepRunner``), and the parts that models are put
together from (``build_mixer`` / ``build_feed_forward``, then ``forward`` on a step's tokens).

``listed`` are the cases by name, ``draw`` gives another one of the same ranges.  A case is run as
a server runs it: weights, cache and step plan are made once (``prepare``), ``run`` is one pass.
Sizes are those of the benchmark's models: Llama in its TinyLlama-1.1B, Llama-2-7B and Llama-3-8B
shapes, and the Sebilorn, Bizetar and Vomotar layers at TinyLlama's width.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

DEVICE = "cuda:0"
PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
# width, feed-forward, query heads, key/value heads, head size, rotation base
LLAMA = {"tinyllama": (2048, 5632, 32, 4, 64, 10000.0),
         "llama2_7b": (4096, 11008, 32, 32, 128, 10000.0),
         "llama3_8b": (4096, 14336, 32, 8, 128, 500000.0)}
VOCABULARY, EPS = 32000, 1e-5


def listed() -> list[dict]:
    return [
        # the headline: a decode step of a whole model, eight requests behind 512-token prompts
        {"name": "decode_b8", "kind": "decode", "dtype": "bf16", "layers": 22, "batch": 8,
         "context": 520},
        # the same step in the true 32-bit mode, the reference's own precision
        {"name": "decode_b8_f32", "kind": "decode", "dtype": "f32", "layers": 22, "batch": 8,
         "context": 520},
        # a long prompt through one attention layer
        {"name": "attention_prompt", "kind": "attention", "dtype": "bf16", "shape": "tinyllama",
         "seqs": 1, "tokens": 2048, "context": 0},
        # many requests with long contexts decode one token each: the cache is what is read
        {"name": "attention_decode_long", "kind": "attention", "dtype": "bf16",
         "shape": "llama3_8b", "seqs": 64, "tokens": 1, "context": 4096},
        # the smallest call: one token of a single request through a feed-forward
        {"name": "mlp_one_token", "kind": "mlp", "dtype": "bf16", "shape": "llama2_7b",
         "tokens": 1},
        # a mixed step: a prompt portion beside decoded tokens, an odd number of rows
        {"name": "mlp_mixed_step", "kind": "mlp", "dtype": "bf16", "shape": "llama2_7b",
         "tokens": 301},
        # a prompt portion through a feed-forward in 32-bit
        {"name": "mlp_prompt_f32", "kind": "mlp", "dtype": "f32", "shape": "tinyllama",
         "tokens": 1000},
        # a long prompt through an attention layer with a window, kept first tokens and a soft cap
        {"name": "window_prompt", "kind": "window", "dtype": "bf16", "seqs": 1, "tokens": 2048,
         "context": 0, "heads": 16, "kv_heads": 4, "dim": 128, "form": "window"},
        # two ragged prompts through sink attention with its convolution, norms and gate
        {"name": "sink_prompts", "kind": "sink", "dtype": "bf16", "seqs": 2, "tokens": 1201,
         "context": 0, "heads": 16, "kv_heads": 4, "dim": 128, "form": "conv"},
        # a decode step of 64 requests through sink attention with distance slopes
        {"name": "sink_decode", "kind": "sink", "dtype": "bf16", "seqs": 64, "tokens": 1,
         "context": 700, "heads": 16, "kv_heads": 4, "dim": 128, "form": "slopes"},
        # a long prompt through a layer of the gated delta rule
        {"name": "delta_prompt", "kind": "delta", "dtype": "bf16", "seqs": 1, "tokens": 2048,
         "heads": 16, "dim": 128},
        # a long prompt through a layer of lightning attention
        {"name": "lightning_prompt", "kind": "lightning", "dtype": "bf16", "seqs": 1,
         "tokens": 2048, "heads": 16, "dim": 128},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "attention", "mlp", "mlp", "window", "sink", "delta", "lightning"])
    dtype = rng.choice(["bf16", "bf16", "f32"])
    wide = dtype == "f32"
    if kind == "decode":
        return {"kind": kind, "dtype": dtype, "layers": rng.randint(2, 8 if wide else 22),
                "batch": _log(rng, 1, 48 if wide else 64), "context": _log(rng, 64, 1900)}
    if kind == "mlp":
        shape = "tinyllama" if wide else rng.choice(sorted(LLAMA))
        return {"kind": kind, "dtype": dtype, "shape": shape,
                "tokens": _log(rng, 1, 1000 if wide else 2048)}
    decode = rng.random() < 0.35
    seqs = _log(rng, 1, 64 if decode else 4)
    tokens = 1 if decode else _log(rng, 9, (400 if wide else 2048) // seqs)
    context = _log(rng, 33, 1900) if decode or rng.random() < 0.3 else 0
    if kind == "attention":
        return {"kind": kind, "dtype": dtype, "shape": rng.choice(sorted(LLAMA)), "seqs": seqs,
                "tokens": tokens, "context": context}
    heads = rng.choice([8, 12, 16])
    dim = rng.choice([64, 128])
    if kind in ("window", "sink"):
        return {"kind": kind, "dtype": dtype, "seqs": seqs, "tokens": tokens, "context": context,
                "heads": heads, "kv_heads": rng.choice([2, 4]), "dim": dim,
                "form": rng.choice(["window", "gated"] if kind == "window" else ["conv", "slopes"])}
    return {"kind": kind, "dtype": dtype, "seqs": seqs, "tokens": tokens, "heads": heads,
            "dim": dim}


# ----------------------------------------------------------------------------- inputs
def _lengths(case) -> "tuple[list[int], list[int]]":
    """(new tokens, tokens already in the cache) of every sequence; ragged."""
    seqs, tokens, context = case["seqs"], case["tokens"], case.get("context", 0)
    new = [max(1, tokens - (i * 29) % (tokens // 3 + 1)) for i in range(seqs)]
    old = [context - (i * 37) % (context // 4 + 1) for i in range(seqs)]
    return new, old


class _Draws:
    """Seeded values on the GPU, the same ones in the same order for ``prepare`` and ``exact``."""

    def __init__(self, case, seed: int) -> None:
        self.dtype = DTYPES[case["dtype"]]
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(1000003 * int(seed) + 17)

    def normal(self, *shape, std=1.0, dtype=None):
        x = torch.randn(shape, generator=self.gen, device=DEVICE)
        return (x * std).to(dtype or self.dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.gen, device=DEVICE) * (hi - lo) + lo


def _shape(case):
    if case["kind"] in ("decode", "attention", "mlp"):
        return LLAMA[case.get("shape", "tinyllama")]
    return None


def _part(case):
    """(kind of the registry, its parameters) of the part that the case runs."""
    kind = case["kind"]
    if kind == "mlp":
        width, inner, *_ = _shape(case)
        return "gated_mlp", dict(width=width, inner=inner, activation="silu")
    if kind == "attention":
        width, _, heads, kv_heads, dim, theta = _shape(case)
        return "attention", dict(width=width, heads=heads, kv_heads=kv_heads, head_dim=dim,
                                 scale=dim ** -0.5, window=None, theta=theta)
    width = LLAMA["tinyllama"][0]
    if kind == "lightning":
        return "lightning_attention", dict(width=width, heads=case["heads"], key_dim=case["dim"],
                                           value_dim=case["dim"], eps=EPS, decay=tuple(
                                               1.0 - 2.0 ** -(4 + i % 8)
                                               for i in range(case["heads"])))
    if kind == "delta":
        return "gated_delta_rule", dict(width=width, heads=case["heads"], kv_heads=case["heads"],
                                        key_dim=case["dim"], value_dim=case["dim"], taps=4,
                                        rank=64, eps=EPS)
    common = dict(width=width, heads=case["heads"], kv_heads=case["kv_heads"],
                  key_dim=case["dim"], value_dim=case["dim"], scale=case["dim"] ** -0.5)
    if kind == "window":
        if case["form"] == "window":
            return "window_attention", dict(common, rotary_dim=case["dim"], theta=500000.0,
                                            scaling=(8.0, 1.0, 4.0, 8192.0), window=1024,
                                            keep_first=4, softcap=30.0, rotate_values=True)
        return "window_attention", dict(common, rotary_dim=64, theta=10000.0, gated=True)
    if case["form"] == "conv":
        return "sink_attention", dict(common, eps=EPS, biased=True, taps=3, norm="head",
                                      gate="feature", adjacent=True, rotary_dim=case["dim"],
                                      theta=100000.0)
    return "sink_attention", dict(common, eps=EPS, norm="whole", slopes=True, gate="head",
                                  temperature=(0.3, 256))


def _weights(case, shapes, draws) -> dict:
    """Random tensors of a part, in the names' order: matrices like a trained model's in size,
    norm weights around one, decay rates over the range such layers are initialised with."""
    out = {}
    for name in sorted(shapes):
        shape, kind = shapes[name]
        if name == "A_log":
            out[name] = draws.uniform(*shape, lo=1.0, hi=16.0).log()
        elif name == "dt_bias":
            out[name] = draws.uniform(*shape, lo=math.log(1e-3), hi=math.log(0.1)).exp().expm1().log()
        elif name.endswith(".conv"):
            out[name] = draws.uniform(*shape, lo=-0.6, hi=0.6)
        elif kind == "matrix":
            out[name] = draws.normal(*shape, std=0.02)
        elif "norm" in name or name == "weight":
            out[name] = draws.uniform(*shape, lo=0.5, hi=1.5)
        else:
            out[name] = draws.normal(*shape, std=0.3, dtype=torch.float32)
    return out


def _pages_of(lengths) -> list[int]:
    return [(n + PAGE - 1) // PAGE for n in lengths]


class _OnePart:
    """What ``StepRunner`` asks of a model, around a single part: it plans the step and keeps the
    step's context, on which the part is then run."""

    def __init__(self, part, width: int) -> None:
        self.part, self.dtype, self.device = part, part.dtype, torch.device(DEVICE)
        self.config = SimpleNamespace(vocabulary=VOCABULARY, width=width)
        self.ctx = None

    def prepare(self, prep) -> None:
        self.part.prepare(prep)

    def forward(self, ctx, bindings):
        self.ctx = ctx


def _admit(cache, new, old, draws) -> list[str]:
    """Requests with ``old`` tokens in the cache and pages for ``new`` more."""
    names = [f"r{i}" for i in range(len(new))]
    for name, n in zip(names, old):
        cache.admit(name)
        if n:
            cache.reserve([(name, n)])
            cache.commit(name, n)
    cache.flush_tables()
    return names


def _cached_rows(binding, cache, names, old, keys, values) -> None:
    """Lay ``keys`` / ``values`` [pages of all requests in order, kv heads, page, dim] into the
    pages that the requests hold."""
    table, ids = binding.block_table, []
    for name, pages in zip(names, _pages_of(old)):
        ids.append(table[cache.slot(name), :pages])
    ids = torch.cat(ids).long()
    held = ids >= 0                 # (the pages that a window has passed are gone)
    binding.k_pages[ids[held]] = keys[held]
    binding.v_pages[ids[held]] = values[held]


def prepare(case, seed):
    from distengine_b200.cache import CacheManager
    from distengine_b200.config.model import PartSpec
    from distengine_b200.engine.step import StepEntry, StepRunner
    from distengine_b200.parts import build_feed_forward, build_mixer
    if case["kind"] == "decode":
        return _prepare_decode(case, seed)
    draws, device = _Draws(case, seed), torch.device(DEVICE)
    kind, params = _part(case)
    width = params["width"]
    if kind == "gated_mlp":
        part = build_feed_forward(PartSpec.of(kind, **params), draws.dtype, device)
        new, old = [case["tokens"]], [0]
    else:
        if kind == "attention":
            params["position"] = PartSpec.of("rope", rotary_dim=params["head_dim"],
                                             theta=params.pop("theta"))
        part = build_mixer(PartSpec.of(kind, **params), draws.dtype, device)
        new, old = _lengths(case)
        if kind in ("gated_delta_rule", "lightning_attention"):
            old = [0] * len(new)
    part.load(_weights(case, part.tensors(), draws))
    x = draws.normal(sum(new), width)
    spec = None if kind == "gated_mlp" else part.cache_spec()
    total = [n + o for n, o in zip(new, old)]
    cache = CacheManager([spec], [None], PAGE, sum(_pages_of(total)) + len(total), len(new),
                         max(total) + PAGE, draws.dtype, device)
    model = _OnePart(part, width)
    runner = StepRunner(model, cache)
    names = _admit(cache, new, old, draws)
    binding = cache.bindings()[0]
    pages, state = binding, None
    if binding is not None and binding.kind == "parts":
        pages, state = binding.parts
    elif binding is not None and binding.kind == "state":
        pages, state = None, binding
    if pages is not None and sum(old):
        count = sum(_pages_of(old))
        keys = draws.normal(count, *pages.k_pages.shape[1:])
        values = draws.normal(count, *pages.v_pages.shape[1:])
        _cached_rows(pages, cache, names, old, keys, values)
    if state is not None and pages is not None:             # a convolution's kept rows
        slots = torch.tensor([cache.slot(n) for n in names], device=device)
        state.state[slots] = draws.normal(len(names), state.state.shape[1], dtype=torch.float32)
    runner.step([StepEntry(name, [0] * n, []) for name, n in zip(names, new)])
    # what a pass leaves in the cache: a prompt's keys and values, a state
    keep = [pages.k_pages, pages.v_pages] if pages is not None and not sum(old) else []
    keep += [state.state] if state is not None else []
    return SimpleNamespace(kind=case["kind"], part=part, ctx=model.ctx, binding=binding, x=x,
                           updated=keep, runner=runner)


def run(state):
    if state.kind == "decode":
        # a decode step that is taken back: the next pass runs the same one
        prepared = state.runner.prepare(state.entries)
        logits = state.runner.launch(prepared, tentative=True)
        for name in state.names:
            state.cache.rewind(name)
        return logits
    if state.kind == "mlp":
        return state.part.forward(state.x, state.ctx)
    # a layer's output, and what it leaves in the cache
    return [state.part.forward(state.x, state.ctx, state.binding), *state.updated]


# ----------------------------------------------------------------------------- a whole model
def _config(case) -> dict:
    width, inner, heads, kv_heads, dim, theta = LLAMA["tinyllama"]
    return {"architectures": ["LlamaForCausalLM"], "vocab_size": VOCABULARY, "hidden_size": width,
            "intermediate_size": inner, "num_hidden_layers": case["layers"],
            "num_attention_heads": heads, "num_key_value_heads": kv_heads, "head_dim": dim,
            "hidden_act": "silu", "rms_norm_eps": EPS, "rope_theta": theta,
            "max_position_embeddings": 2048, "tie_word_embeddings": False}


def _model_tensors(case, draws) -> dict:
    width, inner, heads, kv_heads, dim, _ = LLAMA["tinyllama"]
    q, kv = heads * dim, kv_heads * dim
    out = {"model.embed_tokens.weight": draws.normal(VOCABULARY, width),
           "lm_head.weight": draws.normal(VOCABULARY, width, std=0.02),
           "model.norm.weight": draws.uniform(width, lo=0.5, hi=1.5).to(draws.dtype)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (q, width)), ("self_attn.k_proj", (kv, width)),
                            ("self_attn.v_proj", (kv, width)), ("self_attn.o_proj", (width, q)),
                            ("mlp.gate_proj", (inner, width)), ("mlp.up_proj", (inner, width)),
                            ("mlp.down_proj", (width, inner))):
            out[p + name + ".weight"] = draws.normal(*shape, std=0.02)
        for name in ("input_layernorm", "post_attention_layernorm"):
            out[p + name + ".weight"] = draws.uniform(width, lo=0.5, hi=1.5).to(draws.dtype)
    return out


def _decode_inputs(case, draws):
    """(contexts, token ids, the cached keys and values of every layer in logical pages)."""
    _, _, _, kv_heads, dim, _ = LLAMA["tinyllama"]
    context = case["context"]
    old = [context - (i * 37) % (context // 4 + 1) for i in range(case["batch"])]
    tokens = torch.randint(0, VOCABULARY, (case["batch"],), generator=draws.gen, device=DEVICE)
    count = sum(_pages_of(old))
    cached = [(draws.normal(count, kv_heads, PAGE, dim), draws.normal(count, kv_heads, PAGE, dim))
              for _ in range(case["layers"])]
    return old, tokens.tolist(), cached


def _prepare_decode(case, seed):
    from distengine_b200.cache import CacheManager
    from distengine_b200.config import LlamaConfig
    from distengine_b200.engine.step import StepEntry, StepRunner
    from distengine_b200.models.decoder import DecoderModel
    draws = _Draws(case, seed)
    model = DecoderModel(LlamaConfig.from_json(_config(case)), draws.dtype, DEVICE)
    model.load(_model_tensors(case, draws))
    old, tokens, cached = _decode_inputs(case, draws)
    cache = CacheManager(model.cache_specs(), [e.reads_cache_of for e in model.plan], PAGE,
                         sum(_pages_of([n + 1 for n in old])) + 1, case["batch"], 2048,
                         draws.dtype, DEVICE)
    names = _admit(cache, [1] * len(old), old, draws)
    for binding, (keys, values) in zip(cache.bindings(), cached):
        _cached_rows(binding, cache, names, old, keys, values)
    entries = [StepEntry(name, [t], [0]) for name, t in zip(names, tokens)]
    state = SimpleNamespace(kind="decode", model=model, cache=cache, names=names, entries=entries,
                            runner=StepRunner(model, cache, use_graphs=True))
    for _ in range(3):              # a serving program has decoded before: the step is a graph now
        run(state)
    return state


# ----------------------------------------------------------------------------- work
def _keys_seen(case, params) -> float:
    """Pairs of a query and a key that it sees, over all sequences."""
    new, old = _lengths(case)
    window = params.get("window")
    pairs = 0
    for n, o in zip(new, old):
        if window is None:
            pairs += n * o + n * (n + 1) // 2
        else:
            pairs += sum(min(o + i + 1, window + 4) for i in range(n))
    return float(pairs)


def work(case):
    size = 2 if case["dtype"] == "bf16" else 4
    if case["kind"] == "decode":
        width, inner, heads, kv_heads, dim, _ = LLAMA["tinyllama"]
        weights = case["layers"] * (2 * heads * dim * width + 2 * kv_heads * dim * width
                                    + 3 * inner * width) + VOCABULARY * width
        batch, context = case["batch"], case["context"]
        keys = sum(context - (i * 37) % (context // 4 + 1) for i in range(batch))
        return {"bytes": size * (weights + batch * width
                                 + case["layers"] * 2 * kv_heads * dim * (keys + batch))
                + 4 * batch * VOCABULARY,
                "flops": 2 * weights * batch + case["layers"] * 4 * heads * dim * (keys + batch)}
    _, p = _part(case)
    width = p["width"]
    if case["kind"] == "mlp":
        n, weights = case["tokens"], 3 * width * p["inner"]
        return {"bytes": size * (weights + 2 * n * width), "flops": 2 * weights * n}
    new, old = _lengths(case)
    n = sum(new)
    if case["kind"] in ("delta", "lightning"):
        H, d = p["heads"], p["key_dim"]
        weights = 4 * H * d * width + (H * d * width if case["kind"] == "lightning" else
                                       (H + 2 * 64) * width + 2 * 64 * H * d)
        per_token = (6 if case["kind"] == "delta" else 4) * H * d * d
        return {"bytes": size * (weights + 2 * n * width) + 8 * len(new) * H * d * d,
                "flops": 2 * weights * n + per_token * n}
    H, G = p["heads"], p["kv_heads"]
    d = p.get("key_dim", p.get("head_dim"))
    weights = (2 * H + 2 * G) * d * width
    gate = {"sink/conv": H * d, "sink/slopes": H, "window/gated": H * d}.get(
        f"{case['kind']}/{case.get('form')}", 0)
    weights += gate * width
    keys = sum((o if p.get("window") is None else min(o, p["window"] + 4)) for o in old) + 2 * n
    return {"bytes": size * (weights + 2 * n * width + 2 * G * d * keys),
            "flops": 2 * weights * n + 4 * H * d * _keys_seen(case, p)}


def tolerance(case):
    # about four times what was measured against the 64-bit results: 1e-6 to 6e-6 in 32-bit; in
    # bfloat16 3e-3 to 4e-3 for a layer, 1.3e-2 for the logits behind 22 layers
    if case["dtype"] == "f32":
        return {"rel": 2e-5}
    return {"rel": 3e-2 if case["kind"] == "decode" else 1.2e-2}


# ----------------------------------------------------------------------------- 64-bit results
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _angles(pos, freq):
    a = pos.double()[:, None, None] * freq[None, None, :]
    return torch.cos(a), torch.sin(a)


def _turn(x, pos, freq, sign=1.0, adjacent=False):
    """x [T, heads, d]: pairs (i, i + n) of the first 2n features (or neighbours) turned."""
    n = freq.shape[0]
    c, s = _angles(pos, freq)
    s = sign * s
    if adjacent:
        a, b = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        out = x.clone()
        out[..., 0:2 * n:2], out[..., 1:2 * n:2] = a * c - b * s, b * c + a * s
        return out
    a, b = x[..., :n], x[..., n:2 * n]
    return torch.cat((a * c - b * s, b * c + a * s, x[..., 2 * n:]), -1)


def _frequencies(theta, dims, scaling=None):
    f = float(theta) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)
    if scaling is not None:
        factor, low, high, original = scaling
        wave = 2.0 * math.pi / f
        s = (original / wave - low) / (high - low)
        f = torch.where(wave < original / high, f, torch.where(
            wave > original / low, f / factor, (1.0 - s) * f / factor + s * f))
    return f


def _attend(q, k, v, pos, scale, window=None, keep=0, softcap=None, slopes=None, sink=None):
    """q [T, H, d] at positions ``pos``, keys and values [L, G, d] from position 0 on."""
    H, G = q.shape[1], k.shape[1]
    j = torch.arange(k.shape[0], device=DEVICE)
    dist = pos[:, None] - j[None, :]
    seen = dist >= 0
    if window is not None:
        seen &= (dist < window) | (j < keep)[None, :]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=q.dtype, device=DEVICE)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].t()) * scale
        if slopes is not None:
            s = s - slopes[h] * dist
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~seen, -math.inf)
        top = s.amax(1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        total = e.sum(1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out[:, h] = (e / total) @ v[:, h * G // H]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _dense(pages, table, n):
    """The first n rows [n, kv heads, d] of a request from its logical pages."""
    return pages[table].transpose(1, 2).flatten(0, 1)[:n].double()


def _exact_attention(case, kind, p, w, x, new, old, keys, values, kept):
    H, G = p["heads"], p["kv_heads"]
    d = p.get("key_dim", p.get("head_dim"))
    names = (("q", "k", "v", "o") if kind != "attention" else
             tuple(n + "_proj.weight" for n in ("q", "k", "v", "o")))
    slopes = sink = None
    if p.get("slopes"):
        slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device=DEVICE) / H)
    if kind == "sink_attention":
        sink = w["sink"].double()
    if kind == "window_attention":
        fk, fv = _frequencies(p["theta"], p["rotary_dim"], p.get("scaling")), _frequencies(p["theta"], d)
    elif "theta" in p:
        fk = _frequencies(p["theta"], p.get("rotary_dim", d))
    rows, at, page = [], 0, 0
    for i, (n, o) in enumerate(zip(new, old)):
        h = x[at: at + n].double()
        at += n
        pos = torch.arange(o, o + n, device=DEVICE)
        q, k, v = (h @ w[name].double().t() for name in names[:3])
        if p.get("taps"):
            past = kept[i].double().view(p["taps"] - 1, -1)
            u = torch.cat((q, k, v), 1)
            bias = torch.cat([w[name + ".b"].double() for name in "qkv"])
            taps = torch.cat([w[name + ".conv"].double() for name in "qkv"])
            past = past + bias if o else torch.zeros_like(past)
            u = torch.cat((past, u + bias))
            u = sum(taps[:, j] * u[j: j + n] for j in range(p["taps"]))
            q, k, v = u.split([H * d, G * d, G * d], 1)
        if p.get("norm") == "whole":
            q, k = _rms(q) * w["q.norm"].double(), _rms(k) * w["k.norm"].double()
        if p.get("temperature"):
            coef, every = p["temperature"]
            steps = torch.div(pos + 1, every, rounding_mode="floor").double()
            q = q * (1.0 + coef * torch.log(steps + 1.0))[:, None]
        q, k, v = q.view(n, H, d), k.view(n, G, d), v.view(n, G, d)
        if p.get("norm") == "head":
            q, k = _rms(q) * w["q.norm"].double(), _rms(k) * w["k.norm"].double()
        if "theta" in p:
            q, k = (_turn(t, pos, fk, adjacent=p.get("adjacent", False)) for t in (q, k))
        if p.get("rotate_values"):
            v = _turn(v, pos, fv)
        if o:
            table = list(range(page, page + _pages_of([o])[0]))
            page += len(table)
            k = torch.cat((_dense(keys, table, o), k))
            v = torch.cat((_dense(values, table, o), v))
        out = _attend(q, k, v, pos, p["scale"], p.get("window"), p.get("keep_first", 0),
                      p.get("softcap"), slopes, sink)
        if p.get("rotate_values"):
            out = _turn(out, pos, fv, sign=-1.0)
        if p.get("gate") == "head":
            out = out * torch.sigmoid(h @ w["g"].double().t())[:, :, None]
        out = out.flatten(1)
        if p.get("gate") == "feature" or p.get("gated"):
            out = out * torch.sigmoid(h @ w["g"].double().t())
        rows.append(out @ w[names[3]].double().t())
    return torch.cat(rows)


def _exact_delta(p, w, x, new):
    H, d, at, rows, states = p["heads"], p["key_dim"], 0, [], []
    for n in new:
        h = x[at: at + n].double()
        at += n
        raw = {m: h @ w[m].double().t() for m in "qkv"}
        conv = {}
        for m in "qkv":
            u = torch.cat((raw[m].new_zeros(p["taps"] - 1, raw[m].shape[1]), raw[m]))
            taps = w[m + ".conv"].double()
            conv[m] = _silu(sum(taps[:, j] * u[j: j + n] for j in range(p["taps"]))).view(n, H, d)
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (conv["q"], conv["k"]))
        q, v = q * d ** -0.5, conv["v"]
        beta = torch.sigmoid(h @ w["b"].double().t())
        a = h @ w["a1"].double().t() @ w["a2"].double().t() + w["dt_bias"].double()
        rate = torch.exp(w["A_log"].double())[:, None]
        g = torch.exp(-rate * torch.nn.functional.softplus(a, threshold=1e9).view(n, H, d))
        S = h.new_zeros(H, d, d)
        o = torch.empty_like(v)
        for t in range(n):
            S = S * g[t][:, :, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        gate = torch.sigmoid(h @ w["g1"].double().t() @ w["g2"].double().t()).view(n, H, d)
        rows.append((_rms(o) * w["norm"].double() * gate).flatten(1) @ w["o"].double().t())
        kept = torch.cat([torch.cat((r.new_zeros(p["taps"] - 1, r.shape[1]), r))[n:]
                          for r in (raw[m] for m in "qkv")], 1)
        states.append(torch.cat((S.flatten(), kept.flatten())))
    return [torch.cat(rows), torch.stack(states)]


def _exact_lightning(p, w, x, new):
    H, d, at, rows, states = p["heads"], p["key_dim"], 0, [], []
    decay = torch.tensor(p["decay"], dtype=torch.float64, device=DEVICE)
    for n in new:
        h = x[at: at + n].double()
        at += n
        q, k, v = (_silu(h @ w[m].double().t()).view(n, H, d) for m in "qkv")
        S = h.new_zeros(H, d, d)
        o = torch.empty_like(v)
        for t in range(n):
            S = torch.baddbmm(S * decay[:, None, None], k[t][:, :, None], v[t][:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = _rms(o.flatten(1)) * w["norm"].double() * torch.sigmoid(h @ w["g"].double().t())
        rows.append(o @ w["o"].double().t())
        states.append(S.flatten())
    return [torch.cat(rows), torch.stack(states)]


def _exact_decode(case, seed):
    width, inner, heads, kv_heads, dim, theta = LLAMA["tinyllama"]
    draws = _Draws(case, seed)
    w = _model_tensors(case, draws)
    old, tokens, cached = _decode_inputs(case, draws)
    freq = _frequencies(theta, dim)
    x = w["model.embed_tokens.weight"][tokens].double()
    pos = torch.tensor(old, device=DEVICE)
    for i, (keys, values) in enumerate(cached):
        p = f"model.layers.{i}."
        m = {n: w[p + n + ".weight"].double() for n in (
            "self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
            "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj", "input_layernorm",
            "post_attention_layernorm")}
        h = _rms(x) * m["input_layernorm"]
        q = _turn((h @ m["self_attn.q_proj"].t()).view(-1, heads, dim), pos, freq)
        k = _turn((h @ m["self_attn.k_proj"].t()).view(-1, kv_heads, dim), pos, freq)
        v = (h @ m["self_attn.v_proj"].t()).view(-1, kv_heads, dim)
        out, page = [], 0
        for b, n in enumerate(old):
            table = list(range(page, page + _pages_of([n])[0]))
            page += len(table)
            out.append(_attend(q[b: b + 1], torch.cat((_dense(keys, table, n), k[b: b + 1])),
                               torch.cat((_dense(values, table, n), v[b: b + 1])),
                               pos[b: b + 1], dim ** -0.5))
        x = x + torch.cat(out).flatten(1) @ m["self_attn.o_proj"].t()
        h = _rms(x) * m["post_attention_layernorm"]
        x = x + (_silu(h @ m["mlp.gate_proj"].t()) * (h @ m["mlp.up_proj"].t())) @ m["mlp.down_proj"].t()
    h = _rms(x) * w["model.norm.weight"].double()
    return h @ w["lm_head.weight"].double().t()


def exact(case, seed):
    if case["kind"] == "decode":
        return _exact_decode(case, seed)
    draws = _Draws(case, seed)
    kind, p = _part(case)
    shapes = _tensor_shapes(kind, p)
    w = _weights(case, shapes, draws)
    if kind == "gated_mlp":
        x = draws.normal(case["tokens"], p["width"]).double()
        g, u, d = (w[n + "_proj.weight"].double() for n in ("gate", "up", "down"))
        return (_silu(x @ g.t()) * (x @ u.t())) @ d.t()
    new, old = _lengths(case)
    x = draws.normal(sum(new), p["width"])
    if kind == "gated_delta_rule":
        return _exact_delta(p, w, x, new)
    if kind == "lightning_attention":
        return _exact_lightning(p, w, x, new)
    keys = values = kept = None
    d, G = p.get("key_dim", p.get("head_dim")), p["kv_heads"]
    if sum(old):
        count = sum(_pages_of(old))
        keys, values = (draws.normal(count, G, PAGE, d) for _ in range(2))
    if p.get("taps"):
        kept = draws.normal(len(new), (p["taps"] - 1) * (p["heads"] + 2 * G) * d,
                            dtype=torch.float32)
    out = _exact_attention(case, kind, p, w, x, new, old, keys, values, kept)
    # (the pages' order, and the rows behind a convolution's, are the cache's own)
    return [out] + [None] * ((0 if sum(old) else 2) + (1 if p.get("taps") else 0))


def _tensor_shapes(kind, p) -> dict:
    """Names, shapes and kinds of a part's tensors, as the weight files of such models hold them."""
    width = p["width"]
    if kind == "gated_mlp":
        return {"gate_proj.weight": ((p["inner"], width), "matrix"),
                "up_proj.weight": ((p["inner"], width), "matrix"),
                "down_proj.weight": ((width, p["inner"]), "matrix")}
    H, d = p["heads"], p.get("key_dim", p.get("head_dim"))
    if kind == "gated_delta_rule":
        out = {n: ((H * d, width), "matrix") for n in "qkv"}
        out.update({n + ".conv": ((H * d, p["taps"]), "matrix") for n in "qkv"})
        out.update({"b": ((H, width), "matrix"), "A_log": ((H,), "vector"), "norm": ((d,), "vector"),
                    "a1": ((p["rank"], width), "matrix"), "a2": ((H * d, p["rank"]), "matrix"),
                    "dt_bias": ((H * d,), "vector"), "g1": ((p["rank"], width), "matrix"),
                    "g2": ((H * d, p["rank"]), "matrix"), "o": ((width, H * d), "matrix")})
        return out
    if kind == "lightning_attention":
        out = {n: ((H * d, width), "matrix") for n in "qkvg"}
        out.update({"norm": ((H * d,), "vector"), "o": ((width, H * d), "matrix")})
        return out
    G = p["kv_heads"]
    rows = {"q": H * d, "k": G * d, "v": G * d}
    if kind == "attention":
        return {**{n + "_proj.weight": ((r, width), "matrix") for n, r in rows.items()},
                "o_proj.weight": ((width, H * d), "matrix")}
    out = {n: ((r, width), "matrix") for n, r in rows.items()}
    out["o"] = ((width, H * d), "matrix")
    if p.get("gated"):
        out["g"] = ((H * d, width), "matrix")
    if kind == "sink_attention":
        out["sink"] = ((H,), "bias")
        out["g"] = ((H * d if p["gate"] == "feature" else H, width), "matrix")
        if p.get("biased"):
            out.update({n + ".b": ((r,), "bias") for n, r in rows.items()})
            out.update({n + ".conv": ((r, p["taps"]), "bias") for n, r in rows.items()})
        whole = p["norm"] == "whole"
        out["q.norm"] = (((H * d) if whole else d,), "vector")
        out["k.norm"] = (((G * d) if whole else d,), "vector")
    return out
