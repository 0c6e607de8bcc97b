"""The work that this framework is measured on: single layers, mixers and feed-forwards at the sizes of the repository's own
model shapes, and a short generation through the whole engine.

Every case is built from plain values.  `prepare` makes what a program holds before the call (weights in their parts, the
paged cache with the requests' earlier tokens, the step's context, the layer's input), `run` is one pass through the parts'
own `forward`, or through `Engine.step`.  A step of single tokens is replayed from a CUDA graph, as the engine replays it; a
step with a portion of a prompt is launched kernel by kernel, as the engine launches it.

Kinds:
  layer      one decoder layer (norm, grouped-query attention, norm, gated feed-forward) over a step's rows
  recurrent  one mixer with a state per request: the gated delta rule, gated linear attention, or the delta rule with a decay
             per channel, with its projections and convolutions
  latent     one attention mixer over a compressed latent
  experts    one mixture of experts with a shared expert
  generate   a prompt and then single given tokens through the engine, logits of every step
"""
from __future__ import annotations

import gc
import math

import torch

PAGE = 64
# width, heads, key/value heads, feed-forward: the shapes that bench.py measures (--design-sizes 2048 and 4096, 7b, 14b)
SHAPES = {2048: (16, 4, 8192), 4096: (32, 8, 14336), 3584: (28, 4, 18944), 5120: (40, 8, 13824)}
THETA, EPS = 1e6, 1e-6


def listed():
    return [
        # A user's short question, answered token by token: the smallest calls of all, where launches and latencies count.
        dict(name="generate", kind="generate", width=2048, layers=8, vocab=32000, portion=33, steps=15),
        # Serving a few long conversations: every weight of the layer and 8,192 keys a request for eight tokens.
        dict(name="decode_8x8192", kind="layer", dtype="bfloat16", width=3584, decoders=8, context=8192, portion=0, prefix=0),
        # The first step of a request with a prompt of 2,048 tokens.
        dict(name="prompt_2048", kind="layer", dtype="bfloat16", width=3584, decoders=0, context=0, portion=2048, prefix=0),
        # A busy server: 32 requests decode while a portion of a long prompt is taken in.
        dict(name="mixed_32_512", kind="layer", dtype="bfloat16", width=5120, decoders=32, context=8192, portion=512,
             prefix=3840),
        # The engine in true 32-bit arithmetic, for those who check a model: a prompt, and a few requests decoding.
        dict(name="float32_prompt_300", kind="layer", dtype="float32", width=2048, decoders=0, context=0, portion=300, prefix=0),
        dict(name="float32_decode_4", kind="layer", dtype="float32", width=3584, decoders=4, context=1000, portion=0, prefix=0),
        # Mixers with a state of fixed size, whose point is long prompts: the delta rule and gated linear attention.
        dict(name="delta_prompt_2048", kind="recurrent", mixer="gated_delta", width=2048, decoders=0, portion=2048),
        dict(name="gla_prompt_777", kind="recurrent", mixer="gla", width=4096, decoders=0, portion=777),
        # Attention over a compressed latent: a prompt, and requests decoding (its point: short rows in the cache).
        dict(name="latent_prompt_2048", kind="latent", width=2048, decoders=0, context=0, portion=2048, prefix=0),
        dict(name="latent_decode_8x4096", kind="latent", width=4096, decoders=8, context=4096, portion=0, prefix=0),
        # A mixture of 16 experts of which a token takes two: a decode step (a stream of weights) and a prompt.
        dict(name="experts_decode_8", kind="experts", width=4096, rows=8),
        dict(name="experts_prompt_1000", kind="experts", width=2048, rows=1000),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm of the range."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["generate", "decode", "prompt", "mixed", "float32", "recurrent", "latent", "experts"])
    if kind == "generate":
        return dict(kind="generate", width=2048, layers=rng.randint(2, 8), vocab=32000, portion=_spread(rng, 1, 128),
                    steps=rng.randint(2, 15))
    if kind == "decode":
        b = _spread(rng, 1, 64)
        return dict(kind="layer", dtype="bfloat16", width=rng.choice(sorted(SHAPES)), decoders=b,
                    context=_spread(rng, 16, min(8192, 262144 // b)), portion=0, prefix=0)
    if kind == "prompt":
        return dict(kind="layer", dtype="bfloat16", width=rng.choice(sorted(SHAPES)), decoders=0, context=0,
                    portion=_spread(rng, 17, 2048), prefix=rng.choice([0, _spread(rng, 100, 8192)]))
    if kind == "mixed":
        b = _spread(rng, 1, 32)
        return dict(kind="layer", dtype="bfloat16", width=rng.choice(sorted(SHAPES)), decoders=b,
                    context=_spread(rng, 16, 8192), portion=_spread(rng, 17, 512), prefix=rng.choice([0, _spread(rng, 100, 4096)]))
    if kind == "float32":
        if rng.random() < 0.5:
            return dict(kind="layer", dtype="float32", width=rng.choice([2048, 3584]), decoders=_spread(rng, 1, 8),
                        context=_spread(rng, 16, 2048), portion=0, prefix=0)
        return dict(kind="layer", dtype="float32", width=2048, decoders=0, context=0, portion=_spread(rng, 17, 512),
                    prefix=rng.choice([0, _spread(rng, 16, 512)]))
    if kind == "recurrent":
        mixer = rng.choice(["gated_delta", "gla", "channel_delta"])
        if rng.random() < 0.25:
            return dict(kind="recurrent", mixer=mixer, width=rng.choice([2048, 4096]), decoders=_spread(rng, 1, 32), portion=0)
        return dict(kind="recurrent", mixer=mixer, width=rng.choice([2048, 4096]), decoders=0, portion=_spread(rng, 33, 2048))
    if kind == "latent":
        if rng.random() < 0.5:
            b = _spread(rng, 1, 32)
            return dict(kind="latent", width=rng.choice([2048, 4096]), decoders=b, context=_spread(rng, 16, 8192), portion=0,
                        prefix=0)
        return dict(kind="latent", width=rng.choice([2048, 4096]), decoders=0, context=0, portion=_spread(rng, 33, 2048),
                    prefix=rng.choice([0, _spread(rng, 100, 2048)]))
    return dict(kind="experts", width=rng.choice([2048, 4096]), rows=_spread(rng, 1, 2048))


# ---------------------------------------------------------------------------------------------------------------- inputs
class _Random:
    """Numbers on the GPU from the seed alone, in the order in which they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=self.g).to(dtype)

    def whole(self, n, below):
        return torch.randint(0, below, (n,), generator=self.g, device="cuda").tolist()


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _qwen_layer(r, p, width, dtype):
    """Weights of one decoder layer by their names in a checkpoint."""
    H, K, ff = SHAPES[width]
    d = width // H
    w = {p + "input_layernorm.weight": r.normal(width, std=0.02, mean=1.0, dtype=dtype)}
    for n, rows in (("q", H * d), ("k", K * d), ("v", K * d)):
        w[p + f"self_attn.{n}_proj.weight"] = r.normal(rows, width, std=0.02, dtype=dtype)
        w[p + f"self_attn.{n}_proj.bias"] = r.normal(rows, std=0.02, dtype=dtype)
    w[p + "self_attn.o_proj.weight"] = r.normal(width, H * d, std=0.02, dtype=dtype)
    w[p + "post_attention_layernorm.weight"] = r.normal(width, std=0.02, mean=1.0, dtype=dtype)
    for n, shape in (("gate", (ff, width)), ("up", (ff, width)), ("down", (width, ff))):
        w[p + f"mlp.{n}_proj.weight"] = r.normal(*shape, std=0.02, dtype=dtype)
    return w


def _qwen_config(width, layers, vocab):
    H, K, ff = SHAPES[width]
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "num_hidden_layers": layers, "hidden_size": width,
            "num_attention_heads": H, "num_key_value_heads": K, "intermediate_size": ff, "vocab_size": vocab,
            "max_position_embeddings": 32768, "rope_theta": THETA, "rms_norm_eps": EPS, "tie_word_embeddings": False,
            "sliding_window": 131072, "use_sliding_window": False, "hidden_act": "silu", "max_window_layers": layers}


def _requests(case):
    """(earlier tokens, next tokens) of every request of the step."""
    out = [(case.get("context", 0), 1)] * case["decoders"]
    return out + ([(case.get("prefix", 0), case["portion"])] if case["portion"] else [])


def _layer_inputs(case, seed):
    r, dtype, width = _Random(seed), _dtype(case), case["width"]
    H, K, _ = SHAPES[width]
    weights = _qwen_layer(r, "model.layers.0.", width, dtype)
    # (keys of this size give a softmax that a few dozen keys share)
    past = [(r.normal(K, n, width // H, std=2.0, dtype=dtype), r.normal(K, n, width // H, dtype=dtype))
            for n, _ in _requests(case)]
    h = r.normal(sum(m for _, m in _requests(case)), width)
    return weights, past, h


def _recurrent_sizes(case):
    heads = SHAPES[case["width"]][0]
    if case["mixer"] == "gla":
        return dict(hidden=case["width"], heads=heads // 2, head_dim=128, v_dim=256, tau=16.0, rank=16, eps=1e-5)
    more = dict(decay_rank=128, gate_rank=128) if case["mixer"] == "channel_delta" else {}
    return dict(hidden=case["width"], heads=heads, kv_heads=heads if more else heads // 2, head_dim=128, v_dim=128, conv=4,
                eps=1e-5, **more)


def _recurrent_inputs(case, seed):
    """Weights, the input rows, and per request the state (and the convolutions' last inputs)."""
    r, s, bf = _Random(seed), _recurrent_sizes(case), torch.bfloat16
    E, H, d, dv = s["hidden"], s["heads"], s["head_dim"], s["v_dim"]
    G = s.get("kv_heads", H)
    w = {"q": r.normal(G * d, E, std=0.02, dtype=bf), "k": r.normal(G * d, E, std=0.02, dtype=bf),
         "v": r.normal(H * dv, E, std=0.02, dtype=bf), "o": r.normal(E, H * dv, std=0.02, dtype=bf),
         "norm": r.normal(dv, std=0.02, mean=1.0)}
    if case["mixer"] != "channel_delta":
        w["g"] = r.normal(H * dv, E, std=0.02, dtype=bf)
    if case["mixer"] == "gla":
        w.update({"a1": r.normal(s["rank"], E, std=0.02, dtype=bf), "a2": r.normal(H * d, s["rank"], std=0.3),
                  "a2.b": r.normal(H * d, std=0.02)})
    else:
        for n, rows in (("q", G * d), ("k", G * d), ("v", H * dv)):
            w[n + ".conv"] = r.normal(rows, s["conv"], std=0.3)
        w.update({"b": r.normal(H, E, std=0.02, dtype=bf), "A_log": r.normal(H, std=0.5)})
        if case["mixer"] == "gated_delta":
            w.update({"a": r.normal(H, E, std=0.02, dtype=bf), "dt_bias": r.normal(H, std=0.5, mean=-3.0)})
        else:
            w.update({"dt_bias": r.normal(H * d, std=0.5, mean=-3.0), "a1": r.normal(128, E, std=0.02, dtype=bf),
                      "a2": r.normal(H * d, 128, std=0.1, dtype=bf), "g1": r.normal(128, E, std=0.02, dtype=bf),
                      "g2": r.normal(H * dv, 128, std=0.1, dtype=bf)})
    requests = _requests(case)
    x = r.normal(sum(n for _, n in requests), E, dtype=bf)
    states = [r.normal(len(requests), H, d, dv, std=0.3)]
    if case["mixer"] != "gla":
        states.append(r.normal(len(requests), 2 * G * d + H * dv, s["conv"] - 1))
    return w, x, states


def _latent_sizes(case):
    return dict(hidden=case["width"], heads=SHAPES[case["width"]][0], head_dim=128, rot_dim=64, v_dim=128, kv_rank=512,
                scale=192 ** -0.5, eps=1e-5)


def _latent_inputs(case, seed):
    r, s, bf = _Random(seed), _latent_sizes(case), torch.bfloat16
    E, H, d, rot, dv, R = s["hidden"], s["heads"], s["head_dim"], s["rot_dim"], s["v_dim"], s["kv_rank"]
    w = {"q": r.normal(H * (d + rot), E, std=0.02, dtype=bf), "dkv": r.normal(R + rot, E, std=0.02, dtype=bf),
         "dkv.norm": r.normal(R, std=0.02, mean=1.0), "uk": r.normal(H * d, R, std=0.06, dtype=bf),
         "uv": r.normal(H * dv, R, std=0.06, dtype=bf), "o": r.normal(E, H * dv, std=0.02, dtype=bf)}
    past = [r.normal(n, R + rot, dtype=bf) for n, _ in _requests(case)]
    return w, past, r.normal(sum(n for _, n in _requests(case)), E, dtype=bf)


EXPERTS, TOP = 16, 2


def _experts_sizes(case):
    """Experts a quarter as wide as the dense feed-forward, the shared one half as wide."""
    ff = SHAPES[case["width"]][2]
    return dict(hidden=case["width"], experts=EXPERTS, top=TOP, intermediate=ff // 4, shared_intermediate=ff // 2,
                shared_gate=True, score="sigmoid", renormalize=True, norm_eps=1e-20)


def _experts_inputs(case, seed):
    r, s, bf = _Random(seed), _experts_sizes(case), torch.bfloat16
    E, F, S = s["hidden"], s["intermediate"], s["shared_intermediate"]
    w = {"router": r.normal(EXPERTS, E, std=0.02, dtype=bf), "shared.sg": r.normal(1, E, std=0.02, dtype=bf)}
    for p, f in [(f"e{i}.", F) for i in range(EXPERTS)] + [("shared.", S)]:
        w.update({p + "gate": r.normal(f, E, std=0.02, dtype=bf), p + "up": r.normal(f, E, std=0.02, dtype=bf),
                  p + "down": r.normal(E, f, std=0.02, dtype=bf)})
    return w, r.normal(case["rows"], E, dtype=bf)


def _generate_inputs(case, seed):
    r, width, bf = _Random(seed), case["width"], torch.bfloat16
    w = {"model.embed_tokens.weight": r.normal(case["vocab"], width, dtype=bf),
         "model.norm.weight": r.normal(width, std=0.02, mean=1.0, dtype=bf),
         "lm_head.weight": r.normal(case["vocab"], width, std=0.02, dtype=bf)}
    for i in range(case["layers"]):
        w.update(_qwen_layer(r, f"model.layers.{i}.", width, bf))
    return w, r.whole(case["portion"] + case["steps"], case["vocab"])


# --------------------------------------------------------------------------------------------------------------- prepare
def _runtime(dtype):
    from air_b200.parts.base import Runtime
    return Runtime(device=torch.device("cuda:0"), dtype=dtype, page_tokens=PAGE,
                   status=torch.zeros(1, dtype=torch.int32, device="cuda"))


def _step(case, part, rt, kept=None):
    """The cache of the step's requests at their lengths and the step's context, for a layer or a mixer."""
    from air_b200.cache.manager import CacheManager
    from air_b200.engine.batch import Entry, build_context
    requests = _requests(case)
    pages = sum(-(-(n + m) // PAGE) for n, m in requests)
    cache = CacheManager([part.cache_needs()], PAGE, pages, len(requests), dtype=rt.dtype, device=rt.device,
                         max_blocks=max(-(-(n + m) // PAGE) for n, m in requests))
    for i, (n, _) in enumerate(requests):
        cache.open(i)
        cache.reserve([(i, n)])
        cache.commit(i, n)
    cache.reserve([(i, m) for i, (_, m) in enumerate(requests)])
    planners = {q.plan_key(): q for q in (part.parts() if hasattr(part, "parts") else (part,)) if q.plan_key() is not None}
    ctx = build_context([Entry(i, [0] * m) for i, (_, m) in enumerate(requests)], cache, rt.device, status=rt.status,
                        planners=tuple(planners.values()))
    return cache, ctx


def _into_pages(cache, request, rows):
    """rows [..., n, d] of a request's earlier tokens as whole pages: (page numbers, [pages, ..., PAGE, d])."""
    n = rows.shape[-2]
    full = -(-n // PAGE)
    padded = torch.zeros(rows.shape[:-2] + (full * PAGE, rows.shape[-1]), dtype=rows.dtype, device=rows.device)
    padded[..., :n, :] = rows
    padded = padded.unflatten(-2, (full, PAGE)).movedim(-3, 0)
    return torch.tensor(cache.sequences[request].pages[0][:full], dtype=torch.long, device=rows.device), padded


class _Pass:
    """One pass as a program keeps it: launched kernel by kernel, or for single tokens captured in a CUDA graph.  `states`
    are buffers that a pass advances: the capture's own passes leave them as they were."""

    def __init__(self, call, single_tokens, states=()):
        self.call, self.graph = call, None
        if single_tokens:
            saved = [s.clone() for s in states]
            call()
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            collecting = gc.isenabled()
            gc.disable()              # (another graph must not be freed while this one is captured)
            try:
                with torch.cuda.graph(self.graph):
                    self.outputs = call()
            finally:
                if collecting:
                    gc.enable()
            for s, before in zip(states, saved):
                s.copy_(before)

    def __call__(self):
        if self.graph is None:
            return self.call()
        self.graph.replay()
        return self.outputs


def _prepare_layer(case, seed):
    from air_b200.config import load_config
    from air_b200.engine.model import Model
    from air_b200.parts import registry
    from air_b200.parts.base import Norm
    weights, past, h = _layer_inputs(case, seed)
    width, rt = case["width"], _runtime(_dtype(case))
    config = load_config(_qwen_config(width, 1, 256))
    block = Model(registry.architecture(config.architecture).build_spec(config)).blocks[0]
    block.load(weights, rt)
    del weights
    cache, ctx = _step(case, block, rt)
    views = cache.views(0)
    for i, (k, v) in enumerate(past):
        for which, rows in ((0, k), (1, v)):
            numbers, pages = _into_pages(cache, i, rows)
            views[0].kv[numbers, which] = pages
    cache.flush_tables()
    del past

    def call():
        ctx.shared.clear()
        stream, pending = block.forward(h.clone(), None, ctx, views)
        return {"stream": Norm.add_delta(stream, pending), "pages": views[0].kv}

    return _Pass(call, not case["portion"])


def _mixer(kind, sizes, weights, rt):
    from air_b200.parts import registry
    from air_b200.parts.spec import PartSpec
    part = registry.MIXERS.get(kind)(PartSpec(kind, sizes))
    part.load(weights, rt)
    return part


def _sum_of(delta, rows, width):
    """What a part hands on, added into a stream of zeros as the norm behind it would add it."""
    from air_b200.parts.base import Norm
    return Norm.add_delta(torch.zeros((rows, width), dtype=torch.float32, device="cuda"), delta)


def _prepare_recurrent(case, seed):
    weights, x, states = _recurrent_inputs(case, seed)
    rt = _runtime(torch.bfloat16)
    part = _mixer(case["mixer"], _recurrent_sizes(case), weights, rt)
    cache, ctx = _step(case, part, rt)
    views = cache.views(0)
    slots = [cache.sequences[i].slot for i in range(len(_requests(case)))]
    for view, state in zip(views, states):
        view.state[torch.tensor(slots, device="cuda")] = state
    kept = [view.state for view in views]

    def call():
        ctx.shared.clear()
        return {"out": _sum_of(part.forward(x, ctx, views, True), x.shape[0], case["width"]),
                "states": [k[slots[0]] if len(slots) == 1 else k for k in kept]}

    return _Pass(call, not case["portion"], kept)


def _prepare_latent(case, seed):
    from air_b200.parts.spec import PartSpec
    weights, past, x = _latent_inputs(case, seed)
    rt = _runtime(torch.bfloat16)
    sizes = dict(_latent_sizes(case), position=PartSpec("rope_live", {"rotary_dim": 64, "theta": THETA, "pairing": "half"}))
    part = _mixer("latent_attention", sizes, weights, rt)
    cache, ctx = _step(case, part, rt)
    views = cache.views(0)
    for i, rows in enumerate(past):
        numbers, pages = _into_pages(cache, i, rows)
        views[0].rows[numbers] = pages
    cache.flush_tables()

    def call():
        ctx.shared.clear()
        return {"out": _sum_of(part.forward(x, ctx, views, True), x.shape[0], case["width"]), "rows": views[0].rows}

    return _Pass(call, not case["portion"])


def _prepare_experts(case, seed):
    from types import SimpleNamespace

    from air_b200.parts import registry
    from air_b200.parts.spec import PartSpec
    weights, x = _experts_inputs(case, seed)
    part = registry.FEED_FORWARDS.get("routed_experts")(PartSpec("routed_experts", _experts_sizes(case)))
    part.load(weights, _runtime(torch.bfloat16))
    ctx = SimpleNamespace(residual=None)
    return _Pass(lambda: {"out": _sum_of(part.forward(x, ctx), x.shape[0], case["width"])}, case["rows"] <= 64)


class _Generation:
    """A request through Engine.step: its prompt, then one given token after another; then its pages are free again."""

    def __init__(self, case, seed):
        from air_b200.config import load_config
        from air_b200.engine.engine import Engine, EngineConfig
        from air_b200.engine.model import Model
        from air_b200.parts import registry
        weights, self.tokens = _generate_inputs(case, seed)
        config = load_config(_qwen_config(case["width"], case["layers"], case["vocab"]))
        model = Model(registry.architecture(config.architecture).build_spec(config))
        model.load(weights, _runtime(torch.bfloat16))
        self.prompt = case["portion"]
        self.engine = Engine(model, EngineConfig(page_tokens=PAGE, max_tokens=len(self.tokens) + PAGE, max_requests=1), config)

    def __call__(self):
        from air_b200.engine.batch import Entry
        n = self.prompt
        logits = [self.engine.step([Entry("r", self.tokens[:n], [n - 1])]).clone()]
        for t in self.tokens[n:]:
            logits.append(self.engine.step([Entry("r", [t], [0])]).clone())
        self.engine.finish("r")
        return torch.cat(logits)


_PREPARE = {"layer": _prepare_layer, "recurrent": _prepare_recurrent, "latent": _prepare_latent,
            "experts": _prepare_experts, "generate": _Generation}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state()


# ------------------------------------------------------------------------------------------------------------------ work
def _attention_pairs(requests):
    """Query-key pairs that causal attention over the requests' own keys takes, and keys that are read."""
    return sum(m * n + m * (m + 1) // 2 for n, m in requests), sum(n + m for n, m in requests)


def work(case):
    kind, width = case["kind"], case["width"]
    H, K, ff = SHAPES[width]
    d = width // H
    if kind == "generate":
        per_layer = width * (2 * H * d + 2 * K * d) + 3 * width * ff
        head, n = case["vocab"] * width, case["portion"] + case["steps"]
        calls = 1 + case["steps"]
        pairs = n * (n + 1) // 2
        keys = sum(range(case["portion"], n + 1))
        return {"bytes": calls * 2.0 * (case["layers"] * per_layer + head) + case["layers"] * keys * 4.0 * K * d
                + calls * 4.0 * case["vocab"],
                "flops": 2.0 * (n * case["layers"] * per_layer + calls * head) + 4.0 * case["layers"] * pairs * H * d}
    if kind == "experts":
        T, E, F, S = case["rows"], width, ff // 4, ff // 2
        touched = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** T)
        return {"bytes": 2.0 * (touched * 3 * E * F + 3 * E * S + (EXPERTS + 1) * E) + 2.0 * T * E + 4.0 * T * E,
                "flops": 2.0 * T * (3 * E * (TOP * F + S) + (EXPERTS + 1) * E)}
    requests = _requests(case)
    T = sum(m for _, m in requests)
    if kind == "layer":
        size = 4.0 if case["dtype"] == "float32" else 2.0
        weights = width * (2 * H * d + 2 * K * d) + 3 * width * ff
        pairs, keys = _attention_pairs(requests)
        return {"bytes": size * (weights + 2 * keys * K * d) + 8.0 * T * width,
                "flops": 2.0 * T * weights + 4.0 * pairs * H * d}
    if kind == "latent":
        s = _latent_sizes(case)
        R, rot, hd, dv = s["kv_rank"], s["rot_dim"], s["head_dim"], s["v_dim"]
        weights = width * (H * (hd + rot) + R + rot + H * dv) + H * (hd + dv) * R
        pairs, keys = _attention_pairs(requests)
        # the cheaper of the two orders: keys and values expanded per head, or attention over the latent itself
        expanded = 2.0 * pairs * H * (hd + rot + dv) + 2.0 * keys * H * (hd + dv) * R
        absorbed = 2.0 * pairs * H * (2 * R + rot) + 2.0 * T * H * (hd + dv) * R
        return {"bytes": 2.0 * (weights + keys * (R + rot)) + 2.0 * T * width + 4.0 * T * width,
                "flops": 2.0 * T * (weights - H * (hd + dv) * R) + min(expanded, absorbed)}
    s = _recurrent_sizes(case)
    H, d, dv, G = s["heads"], s["head_dim"], s["v_dim"], s.get("kv_heads", s["heads"])
    weights = width * (2 * G * d + 2 * H * dv)
    if case["mixer"] == "channel_delta":
        weights += 256 * width + 128 * H * (d + dv)
    else:
        weights += width * H * dv
    state = len(requests) * H * d * dv
    return {"bytes": 2.0 * weights + 8.0 * state + 2.0 * T * width + 4.0 * T * width,
            "flops": 2.0 * T * weights + (4.0 if case["mixer"] == "gla" else 6.0) * T * H * d * dv}


# ------------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times the relative error against 64-bit arithmetic that these sizes show.  (32-bit sums: 3e-6 of a layer's
    stream.  bfloat16 rows between the products: 0.002 to 0.005 of a layer, 0.006 of eight layers' logits.)"""
    if case["kind"] == "layer":
        return {"rel": 1.2e-5} if case["dtype"] == "float32" else {"rel": 2e-2}
    return {"rel": {"generate": 2.4e-2, "recurrent": 7e-3, "latent": 1.6e-2, "experts": 1.3e-2}[case["kind"]]}


# ----------------------------------------------------------------------------------------------------------------- exact
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turned(x, positions):
    """x [..., T, r]: element i with i + r / 2, angle position * THETA^(-2i / r)."""
    r = x.shape[-1]
    f = THETA ** (-2.0 * torch.arange(r // 2, dtype=torch.float64, device=x.device) / r)
    a = positions.double()[:, None] * f[None]
    c, s, u, v = torch.cos(a), torch.sin(a), x[..., : r // 2], x[..., r // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], dim=-1)


def _causal(scores, earlier):
    T, n = scores.shape[-2:]
    seen = torch.arange(n, device=scores.device)[None] <= earlier + torch.arange(T, device=scores.device)[:, None]
    return torch.softmax(scores.masked_fill(~seen, -math.inf), dim=-1)


def _exact_layer(w, p, h, requests, past, width):
    """One decoder layer in 64 bits; past: per request (keys [K, n, d], values).  Also the requests' keys and values."""
    H, K, _ = SHAPES[width]
    d = width // H
    f = lambda n: w[p + n].double()  # noqa: E731
    x = _rms(h, f("input_layernorm.weight"), EPS)
    q, k, v = (x @ f(f"self_attn.{n}_proj.weight").t() + f(f"self_attn.{n}_proj.bias") for n in "qkv")
    outs, kept, at = [], [], 0
    for (n, m), (pk, pv) in zip(requests, past):
        pos = torch.arange(n, n + m, device=h.device)
        rows = slice(at, at + m)
        at += m
        heads = lambda y, c: y[rows].view(m, c, d).transpose(0, 1)  # noqa: E731
        kk = torch.cat([pk.double(), _turned(heads(k, K), pos)], dim=1)
        vv = torch.cat([pv.double(), heads(v, K)], dim=1)
        qq = _turned(heads(q, H), pos).view(K, H // K, m, d)
        out = torch.empty((K, H // K, m, d), dtype=torch.float64, device=h.device)
        for g in range(K):
            out[g] = _causal(qq[g] @ kk[g].t() * d ** -0.5, n) @ vv[g]
        outs.append(out.view(H, m, d).transpose(0, 1).reshape(m, H * d))
        kept.append((kk, vv))
    h = h + torch.cat(outs) @ f("self_attn.o_proj.weight").t()
    x = _rms(h, f("post_attention_layernorm.weight"), EPS)
    act = torch.nn.functional.silu(x @ f("mlp.gate_proj.weight").t()) * (x @ f("mlp.up_proj.weight").t())
    return h + act @ f("mlp.down_proj.weight").t(), kept


def _exact_recurrent(case, seed):
    w, x, states = _recurrent_inputs(case, seed)
    s = _recurrent_sizes(case)
    w = {n: t.double() for n, t in w.items()}
    x, H, d, dv = x.double(), s["heads"], s["head_dim"], s["v_dim"]
    G, requests, T = s.get("kv_heads", H), _requests(case), x.shape[0]
    lin = lambda n: x @ w[n].t()  # noqa: E731
    silu, sig = torch.nn.functional.silu, torch.sigmoid
    states, tails, at, beta = [t.double() for t in states], [], 0, None
    rows = []
    for _, m in requests:
        rows.append(slice(at, at + m))
        at += m
    if case["mixer"] == "gla":
        q, k, v = lin("q") * d ** -0.5, lin("k"), lin("v")
        keep = sig(lin("a1") @ w["a2"].t() + w["a2.b"]).pow(1.0 / s["tau"]).view(T, H, d)
        gate = silu(lin("g"))
    else:
        raw, taps = torch.cat([lin("q"), lin("k"), lin("v")], dim=1), s["conv"]
        kernel, y = torch.cat([w[n + ".conv"] for n in "qkv"]), torch.empty_like(raw)
        for i, part in enumerate(rows):
            full = torch.cat([states[1][i].t(), raw[part]])           # (the last inputs, the oldest first)
            n = raw[part].shape[0]
            y[part] = silu(sum(full[j:j + n] * kernel[:, j] for j in range(taps)))
            tails.append(full[-(taps - 1):].t())
        q, k, v = y[:, :G * d], y[:, G * d:2 * G * d], y[:, 2 * G * d:]
        unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = unit(q.reshape(T, G, d)) * d ** -0.5, unit(k.reshape(T, G, d))
        beta, rate = sig(lin("b")), -torch.exp(w["A_log"])
        softplus = lambda z: torch.logaddexp(z, torch.zeros_like(z))  # noqa: E731
        if case["mixer"] == "gated_delta":
            keep = torch.exp(rate * softplus(lin("a") + w["dt_bias"]))[:, :, None].expand(T, H, d)
            gate = silu(lin("g"))
        else:
            z = (lin("a1") @ w["a2"].t() + w["dt_bias"]).view(T, H, d)
            keep, gate = torch.exp(rate[:, None] * softplus(z)), sig(lin("g1") @ w["g2"].t())
        q, k = (z.repeat_interleave(H // G, dim=1) for z in (q, k))
    q, k, v = q.reshape(T, H, d), k.reshape(T, H, d), v.reshape(T, H, dv)
    o = torch.empty((T, H, dv), dtype=torch.float64, device=x.device)
    for i, part in enumerate(rows):
        S = states[0][i].clone()
        for t in range(part.start, part.stop):
            S *= keep[t][:, :, None]
            u = v[t]
            if beta is not None:
                u = beta[t][:, None] * (u - (S * k[t][:, :, None]).sum(1))
            S += k[t][:, :, None] * u[:, None, :]
            o[t] = (S * q[t][:, :, None]).sum(1)
        states[0][i] = S
    out = (_rms(o, w["norm"], s["eps"]).reshape(T, H * dv) * gate) @ w["o"].t()
    if len(requests) > 1:         # (the states lie in the order of the requests' slots, which is the cache's own affair)
        return {"out": out, "states": [None] * len(states)}
    return {"out": out, "states": [states[0][0]] + ([tails[0]] if tails else [])}


def _exact_latent(case, seed):
    w, past, x = _latent_inputs(case, seed)
    s = _latent_sizes(case)
    w, x, R = {n: t.double() for n, t in w.items()}, x.double(), s["kv_rank"]
    H, d, rot, dv = s["heads"], s["head_dim"], s["rot_dim"], s["v_dim"]
    q, both = (x @ w["q"].t()).view(-1, H, d + rot), x @ w["dkv"].t()
    c, outs, at = _rms(both[:, :R], w["dkv.norm"], s["eps"]), [], 0
    for (n, m), rows in zip(_requests(case), past):
        pos, part = torch.arange(n, n + m, device=x.device), slice(at, at + m)
        at += m
        latent = torch.cat([rows[:, :R].double(), c[part]])
        turned = torch.cat([rows[:, R:].double(), _turned(both[part, R:], pos)])
        out = torch.empty((m, H, dv), dtype=torch.float64, device=x.device)
        for h in range(H):
            key, value = latent @ w["uk"][h * d:(h + 1) * d].t(), latent @ w["uv"][h * dv:(h + 1) * dv].t()
            scores = q[part, h, :d] @ key.t() + _turned(q[part, h, d:], pos) @ turned.t()
            out[:, h] = _causal(scores * s["scale"], n) @ value
        outs.append(out.view(m, H * dv))
    return {"out": torch.cat(outs) @ w["o"].t(), "rows": None}


def _exact_experts(case, seed):
    w, x = _experts_inputs(case, seed)
    s = _experts_sizes(case)
    x = x.double()
    expert = lambda p, u: (torch.nn.functional.silu(u @ w[p + "gate"].double().t())  # noqa: E731
                           * (u @ w[p + "up"].double().t())) @ w[p + "down"].double().t()
    scores = torch.sigmoid(x @ w["router"].double().t())
    best, chosen = scores.topk(TOP, dim=1)
    weight = best / (best.sum(1, keepdim=True) + s["norm_eps"])
    out = torch.sigmoid(x @ w["shared.sg"].double().t()) * expert("shared.", x)
    for e in range(EXPERTS):
        token, choice = (chosen == e).nonzero(as_tuple=True)
        if len(token):                  # (a choice's weight multiplies the expert's input)
            out.index_add_(0, token, expert(f"e{e}.", x[token] * weight[token, choice][:, None]))
    return {"out": out}


def _exact_generate(case, seed):
    w, tokens = _generate_inputs(case, seed)
    width, n = case["width"], len(tokens)
    H, K, _ = SHAPES[width]
    h = w["model.embed_tokens.weight"][torch.tensor(tokens, device="cuda")].double()
    none = torch.zeros((K, 0, width // H), dtype=torch.float64, device="cuda")
    for i in range(case["layers"]):
        h, _ = _exact_layer(w, f"model.layers.{i}.", h, [(0, n)], [(none, none)], width)
    h = h[case["portion"] - 1:]
    return _rms(h, w["model.norm.weight"].double(), EPS) @ w["lm_head.weight"].double().t()


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "layer":
            weights, past, h = _layer_inputs(case, seed)
            stream, _ = _exact_layer(weights, "model.layers.0.", h.double(), _requests(case), past, case["width"])
            return {"stream": stream, "pages": None}
        return {"recurrent": _exact_recurrent, "latent": _exact_latent, "experts": _exact_experts,
                "generate": _exact_generate}[case["kind"]](case, seed)
