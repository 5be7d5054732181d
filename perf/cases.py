"""The work a user of this engine has it do, as cases that can be timed and checked.

Sizes are those of the repository's own benchmark shapes (Llama-2-7B, Llama-2-13B and OpenLLaMA-3B
shapes, and the Medolorn design at the 7B layer sizes).  Decode steps run from CUDA graphs, as the
engine runs them; prompt portions are launched step by step, as the engine launches them.

Kinds of case:

* ``model``: whole steps of a decoder of a few layers: batch description, page tables, forward
  (and sampling where tokens are decoded); the result is the logits.
* ``attention``: one attention layer (projection, rotary encoding, cache append, paged attention,
  output projection into the residual) over decoded tokens, prompt portions, or both in one step.
* ``mlp``: one gated feed-forward into the residual.
* ``head``: final norm and output head of the rows that are sampled.
* ``experts``: one routed feed-forward.
* ``delta``: one linear-attention layer (gated delta rule) over prompts.
* ``latent``: one latent-attention layer (one cached row for all heads, sliding window).
"""
import math
import random
import zlib

import torch

from helix_runtime_b200 import LlamaConfig, StepEntry, StepFunction
from helix_runtime_b200.cache.manager import CacheManager
from helix_runtime_b200.config.medolorn import (DeltaMixerConfig, LatentAttentionConfig,
                                                MedolornConfig, MedolornLayerConfig,
                                                RoutedMlpConfig)
from helix_runtime_b200.config.registry import architecture_for
from helix_runtime_b200.engine.graphs import DecodeGraphs, bucketed_context
from helix_runtime_b200.models.decoder import DecoderModel
from helix_runtime_b200.sampling.sampler import Sampler

SHAPES = {
    "llama-2-7b": dict(hidden_size=4096, intermediate_size=11008, num_attention_heads=32,
                       num_key_value_heads=32, head_dim=128, max_position_embeddings=4096,
                       rms_norm_eps=1e-5, rope_theta=10000.0),
    "openllama-3b": dict(hidden_size=3200, intermediate_size=8640, num_attention_heads=32,
                         num_key_value_heads=32, head_dim=100, max_position_embeddings=2048,
                         rms_norm_eps=1e-6, rope_theta=10000.0),
    "llama-2-13b": dict(hidden_size=5120, intermediate_size=13824, num_attention_heads=40,
                        num_key_value_heads=40, head_dim=128, max_position_embeddings=4096,
                        rms_norm_eps=1e-5, rope_theta=10000.0),
}
VOCAB = 32000
PAGE = 16
PORTION = 2048               # tokens of a step
EXPERTS = dict(ff=2816, experts=16, top=4, scale=1.0)
DELTA = dict(heads=32, kv_heads=16, dim=128, vdim=128, conv=4)
LATENT = dict(heads=32, dim=128, rot_dim=64, vdim=128, kv_rank=192, q_rank=1024,
              scale=1.0 / math.sqrt(192.0), window=1024, rot_base=500000.0, rot_dims=64)
MEDOLORN_WIDTH, MEDOLORN_EPS, CANON_TAPS = 4096, 1e-5, 4
DEVICE = "cuda:0"


# ------------------------------------------------------------------------------ the cases

def listed():
    return [
        # a prompt of 2,048 tokens: the time to the first token
        dict(name="model prompt 2048", kind="model", shape="llama-2-7b", layers=4, decode=0,
             low=0, high=0, prompt=2048),
        # the headline: a decode step of eight requests in the middle of their answers
        dict(name="model decode 8", kind="model", shape="llama-2-7b", layers=4, decode=8,
             low=512, high=767, prompt=0),
        # the attention layer of a long prompt
        dict(name="attention prompt 2048", kind="attention", shape="llama-2-7b", decode=0, low=0,
             high=0, portions=1, portion_low=2048, portion_high=2048, behind=0),
        # a full serving batch at contexts of all lengths
        dict(name="attention decode 64", kind="attention", shape="llama-2-7b", decode=64, low=128,
             high=2303, portions=0, portion_low=0, portion_high=0, behind=0),
        # a serving step that interleaves prompt portions with decoding; heads of 100
        dict(name="attention mixed 3b", kind="attention", shape="openllama-3b", decode=32, low=64,
             high=1151, portions=3, portion_low=200, portion_high=512, behind=512),
        # the feed-forward of a prompt whose length is no multiple of a tile, the widest shape
        dict(name="mlp prompt 1900 13b", kind="mlp", shape="llama-2-13b", tokens=1900,
             dtype="bfloat16"),
        # the smallest call: one token's feed-forward, a pure stream of weights
        dict(name="mlp decode 1 3b", kind="mlp", shape="openllama-3b", tokens=1, dtype="bfloat16"),
        # the 32-bit path, a prompt portion
        dict(name="mlp float32 512 3b", kind="mlp", shape="openllama-3b", tokens=512,
             dtype="float32"),
        # the output head of a full serving batch
        dict(name="head 64", kind="head", shape="llama-2-7b", rows=64),
        # routed experts in a prompt portion
        dict(name="experts prompt 1024", kind="experts", tokens=1024),
        # linear attention over two prompts of uneven length
        dict(name="delta prompts 2", kind="delta", requests=2, low=700, high=1024),
        # latent attention over a prompt longer than its window
        dict(name="latent prompt 2048", kind="latent", decode=0, low=0, high=0, portions=1,
             portion_low=2048, portion_high=2048, behind=0),
    ]


def _between(rng, low, high):
    """A whole number, spread over the logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["model", "attention", "attention", "mlp", "mlp", "mlp", "head", "experts",
                       "delta", "latent"])
    if kind == "model":
        if rng.random() < 0.5:
            return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), layers=rng.randint(1, 2),
                        decode=0, low=0, high=0, prompt=_between(rng, 16, 1900))
        low = _between(rng, 32, 900)
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), layers=rng.randint(1, 2),
                    decode=_between(rng, 1, 64), low=low, high=low + _between(rng, 1, 512),
                    prompt=0)
    if kind in ("attention", "latent"):
        case = dict(kind=kind, decode=0, low=0, high=0, portions=0, portion_low=0, portion_high=0,
                    behind=0)
        if kind == "attention":
            case["shape"] = rng.choice(sorted(SHAPES))
        make_up = rng.choice(["decode", "prompt", "mixed"])
        if make_up != "prompt":
            low = _between(rng, 16, 900)
            case.update(decode=_between(rng, 1, 64), low=low, high=low + _between(rng, 1, 1000))
        if make_up != "decode":
            portions = rng.randint(1, 3)
            high = _between(rng, 24, 1900 // portions)
            case.update(portions=portions, portion_low=max(17, high // 2), portion_high=high,
                        behind=rng.choice([0, 0, 256, 777]) if high <= 400 else 0)
        return case
    if kind == "mlp":
        if rng.random() < 0.25:
            return dict(kind=kind, shape="openllama-3b", tokens=_between(rng, 1, 512),
                        dtype="float32")
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), tokens=_between(rng, 1, 2048),
                    dtype="bfloat16")
    if kind == "head":
        return dict(kind=kind, shape=rng.choice(sorted(SHAPES)), rows=_between(rng, 1, 64))
    if kind == "experts":
        return dict(kind=kind, tokens=_between(rng, 1, 2048))
    requests = rng.randint(1, 4)
    high = _between(rng, 64, 2048 // requests)
    return dict(kind=kind, requests=requests, low=max(2, high // 3), high=high)


# ------------------------------------------------------------- inputs, made from the seed alone

def _generator(*words):
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(zlib.crc32("/".join(str(word) for word in words).encode()))
    return generator


def _matrix(name, shape, seed, dtype):
    value = torch.randn(shape, generator=_generator(seed, name), device=DEVICE)
    return value.mul_(0.02).to(dtype)


def _vector(name, shape, seed):
    """Per-channel vectors and small tables, as trained models have them."""
    leaf = name.rsplit(".", 1)[-1]
    if leaf == "A_log":
        return torch.linspace(math.log(1.0 / 16.0), 0.0, shape[0], device=DEVICE)
    if leaf == "dt_bias":
        return torch.full(shape, -2.25, device=DEVICE)
    spread = torch.randn(shape, generator=_generator(seed, name), device=DEVICE) * 0.1
    if leaf == "conv":
        spread[:, -1] += 1.0                         # a filter passes the token itself
    if leaf in ("conv", "canon1", "norm1", "norm2", "b") or name in ("final.norm", "embed.norm"):
        return spread                                # stored around zero
    return 1.0 + spread


def _rows(request, count, width, seed, dtype):
    """What a layer reads: the rows of one request, as they leave a norm."""
    return torch.randn((count, width), generator=_generator(seed, "rows", request),
                       device=DEVICE).to(dtype)


def _tokens(request, count, seed):
    rng = random.Random(f"{seed}/tokens/{request}")
    return [rng.randrange(VOCAB) for _ in range(count)]


def _lengths(case):
    """(cached tokens, new tokens) of every request of the step."""
    kind = case["kind"]
    if kind == "head":
        return [(0, 1)] * case["rows"]
    if kind in ("mlp", "experts"):          # as many requests that decode, or one prompt
        return [(0, 1)] * case["tokens"] if case["tokens"] <= 64 else [(0, case["tokens"])]
    rng = random.Random("|".join(f"{key}={case[key]}" for key in sorted(case) if key != "name"))
    if kind == "delta":
        return [(0, rng.randint(case["low"], case["high"])) for _ in range(case["requests"])]
    if kind == "model" and case["prompt"]:
        return [(0, case["prompt"])]
    lengths = [(rng.randint(case["low"], case["high"]), 1) for _ in range(case["decode"])]
    for index in range(case.get("portions", 0)):
        new = rng.randint(case["portion_low"], case["portion_high"])
        lengths.append((index * case["behind"], new))
    return lengths


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _config(case):
    kind = case["kind"]
    if kind in ("model", "head", "attention", "mlp"):
        vocab = VOCAB if kind in ("model", "head") else 64
        return LlamaConfig(vocab_size=vocab, num_hidden_layers=case.get("layers", 1),
                           **SHAPES[case["shape"]])
    mixer = ("latent_attention", LatentAttentionConfig(**LATENT)) if kind == "latent" else \
        ("delta", DeltaMixerConfig(**DELTA))
    mlp = RoutedMlpConfig(**EXPERTS) if kind == "experts" else None
    return MedolornConfig(vocab=64, width=MEDOLORN_WIDTH, norm_eps=MEDOLORN_EPS,
                          canon_taps=CANON_TAPS, layers=(MedolornLayerConfig(*mixer, mlp),),
                          max_positions=4096)


def _model(case, seed):
    config = _config(case)
    model = DecoderModel(architecture_for(config.to_dict()).build_spec(config))
    dtype = _dtype(case)
    tensors = {}
    for request in model.tensor_requests():
        tensors[request.name] = _vector(request.name, request.shape, seed) \
            if request.role == "scale" else _matrix(request.name, request.shape, seed, dtype)
    model.bind(tensors, dtype, torch.device(DEVICE))
    return model


# ---------------------------------------------------------------------------------- prepare

def _step(model, lengths, capacity):
    kv, state = model.cache_needs()
    pages = sum(-(-(cached + new + 1) // PAGE) for cached, new in lengths)
    cache = CacheManager(kv, state, PAGE, pages, len(lengths), model.max_positions, model.dtype,
                         torch.device(DEVICE))
    step = StepFunction(model, cache, max_tokens=capacity, max_requests=len(lengths))
    for request in range(len(lengths)):
        cache.admit(request)
    return cache, step


def prepare(case, seed):
    with torch.no_grad():
        return _prepare_model(case, seed) if case["kind"] == "model" else \
            _prepare_part(case, seed)


def _prepare_model(case, seed):
    model = _model(case, seed)
    lengths = _lengths(case)
    cache, step = _step(model, lengths, PORTION)
    state = dict(kind="model", model=model, cache=cache, step=step)
    prompts = [_tokens(request, cached + new, seed)
               for request, (cached, new) in enumerate(lengths)]
    if case["prompt"]:
        state["entries"] = [StepEntry(0, prompts[0], [case["prompt"] - 1])]
        cache.release(0)
        return state
    for request, (cached, _) in enumerate(lengths):
        step.run([StepEntry(request, prompts[request][:cached], [])])
    state["entries"] = [StepEntry(request, prompts[request][-1:], [0])
                        for request in range(len(lengths))]
    state["context"] = bucketed_context(max(cached + 1 for cached, _ in lengths))
    state["graphs"] = DecodeGraphs(step, Sampler(torch.device(DEVICE), len(lengths)))
    for _ in range(3):       # the engine records a step that has come up three times
        run(state)
    return state


def _prepare_part(case, seed):
    model = _model(case, seed)
    dtype, kind, width = model.dtype, case["kind"], model.hidden_size
    lengths = _lengths(case)
    n = sum(new for _, new in lengths)
    cache, step = _step(model, lengths, PORTION + 64)
    x = torch.zeros((step.max_tokens, width), dtype=dtype, device=DEVICE)
    residual = torch.zeros((step.max_tokens, width), dtype=torch.float32, device=DEVICE)
    view = model.layer_cache(cache, 0)
    state = dict(kind=kind, model=model, step=step, view=view, x=x, residual=residual, n=n)
    fresh = []
    for request, (cached, new) in enumerate(lengths):
        rows = _rows(request, cached + new, width, seed, dtype)
        for start in range(0, cached, PORTION):      # what earlier steps left in the cache
            count = min(PORTION, cached - start)
            entries = [StepEntry(request, [0] * count, [])]
            ctx, _, _, new_lengths = step.prepare(entries)
            x[:count] = rows[start:start + count]
            model.blocks[0].mixer.forward(ctx, view, x, residual)
            step.finish(entries, new_lengths, ctx)
        fresh.append(rows[cached:].clone())
    x[:n] = torch.cat(fresh)
    state["before"] = torch.randn((n, width), generator=_generator(seed, "residual"),
                                  device=DEVICE)
    state["ctx"] = step.prepare([StepEntry(request, [0] * new, [])
                                 for request, (_, new) in enumerate(lengths)])[0]
    if kind == "head":
        state["rows"] = torch.arange(n - 1, -1, -1, dtype=torch.int32, device=DEVICE)
        state["wanted"] = torch.zeros_like(x)
        state["logits"] = torch.zeros((n, VOCAB), dtype=torch.float32, device=DEVICE)
    if all(new == 1 for _, new in lengths):          # a decode step: recorded and replayed
        for _ in range(2):
            _layer(state)
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            _layer(state)
    return state


# -------------------------------------------------------------------------------------- run

def _layer(state):
    ctx, kind, n, model = state["ctx"], state["kind"], state["n"], state["model"]
    if kind == "head":
        model.final_norm.forward(ctx, state["before"], state["wanted"], rows=state["rows"],
                                 n_rows=n)
        model.lm_head.forward(ctx, state["wanted"], state["logits"], n)
        return
    residual, block = state["residual"], model.blocks[0]
    residual[:n].copy_(state["before"])
    if kind in ("mlp", "experts"):
        block.feed_forward.forward(ctx, state["x"], residual)
        return
    if state["view"].state is not None and kind == "delta":
        state["view"].state.zero_()          # admission gives a request zeroed state
    block.mixer.forward(ctx, state["view"], state["x"], residual)


def _model_step(state):
    cache, step, entries = state["cache"], state["step"], state["entries"]
    if "graphs" not in state:                # a prompt: admitted, run, its first logits read
        cache.admit(0)
        logits = step.run(entries, check_status=False)
        cache.release(0)
        return logits
    ctx, want_rows, n_want, _ = step.prepare(entries, context_hint=state["context"])
    state["graphs"].run(ctx, want_rows, n_want, True)
    for entry in entries:                    # nothing is kept: the next pass decodes here again
        cache.rollback(entry.request)
    return ctx.workspace.get("model.logits", (ctx.capacity, VOCAB), torch.float32)[:n_want]


def run(state):
    with torch.no_grad():
        if state["kind"] == "model":
            return _model_step(state)
        if "graph" in state:
            state["graph"].replay()
        else:
            _layer(state)
        if state["kind"] == "head":
            return state["logits"]
        out = {"residual": state["residual"][:state["n"]]}
        view = state["view"]
        if state["kind"] in ("attention", "latent"):
            out.update(keys=view.keys, values=view.values)
        if state["kind"] == "delta":
            out["state"] = view.state
        return out


# ------------------------------------------------------------------------------------- work

def _attended(lengths, window=None):
    """Pairs of a query and a key it sees, and cached rows that are read."""
    pairs = rows = 0
    for cached, new in lengths:
        for place in range(cached, cached + new):
            pairs += min(place + 1, window or place + 1)
        rows += min(cached, window + new) if window else cached
    return pairs, rows


def work(case):
    kind, size = case["kind"], 4 if case.get("dtype") == "float32" else 2
    lengths = _lengths(case)
    n = sum(new for _, new in lengths)
    if kind in ("model", "head", "attention", "mlp"):
        shape = SHAPES[case["shape"]]
        h, i = shape["hidden_size"], shape["intermediate_size"]
        q = shape["num_attention_heads"] * shape["head_dim"]
    else:
        h = MEDOLORN_WIDTH
    if kind == "mlp":
        return {"bytes": 3 * h * i * size + n * h * (size + 8), "flops": 6 * n * h * i}
    if kind == "head":
        return {"bytes": VOCAB * h * 2 + n * (h * 4 + VOCAB * 4), "flops": 2 * n * h * VOCAB}
    if kind == "experts":
        ff, e, top = EXPERTS["ff"], EXPERTS["experts"], EXPERTS["top"]
        used = e * (1.0 - (1.0 - top / e) ** n)
        return {"bytes": int(used * 3 * h * ff * 2 + e * h * 2 + n * h * 10),
                "flops": n * (6 * top * h * ff + 2 * e * h)}
    if kind == "delta":
        heads, vd = DELTA["heads"], DELTA["heads"] * DELTA["vdim"]
        qk = DELTA["kv_heads"] * DELTA["dim"]
        weights = h * (2 * qk + 3 * vd + 2 * heads)
        state = len(lengths) * heads * DELTA["dim"] * DELTA["vdim"] * 4
        return {"bytes": weights * 2 + n * h * 10 + state,
                "flops": 2 * n * weights + 6 * n * heads * DELTA["dim"] * DELTA["vdim"]}
    if kind == "latent":
        heads, dim, rot, vd = LATENT["heads"], LATENT["dim"], LATENT["rot_dim"], LATENT["vdim"]
        rank, qr = LATENT["kv_rank"], LATENT["q_rank"]
        pairs, rows = _attended(lengths, LATENT["window"])
        weights = h * (qr + rank + rot) + qr * heads * (dim + rot) + heads * (dim + vd) * rank \
            + 2 * h * heads * vd
        return {"bytes": weights * 2 + n * h * 10 + (rows + n) * (rank + rot) * 2,
                "flops": 2 * n * weights + 2 * pairs * heads * (dim + rot + vd)}
    pairs, rows = _attended(lengths)
    layer = 4 * h * q
    if kind == "attention":
        return {"bytes": layer * 2 + n * h * 10 + (rows + n) * 2 * q * 2,
                "flops": 2 * n * layer + 4 * pairs * q}
    layers, wanted = case["layers"], case["decode"] or 1
    return {"bytes": layers * (layer * 2 + 3 * h * i * 2 + (rows + n) * 2 * q * 2) + VOCAB * h * 2
            + n * h * 2 + wanted * VOCAB * 4,
            "flops": layers * (2 * n * layer + 4 * pairs * q + 6 * n * h * i)
            + 2 * wanted * h * VOCAB}


def tolerance(case):
    # 32 bits: the order of the sums.  bfloat16: the roundings between a layer's kernels, which
    # two correct orders of the float32 sums do not always take alike; measured against 64 bits
    # 0.0013 (attention), 0.0016 (feed-forward, head), 0.0008 (experts), 0.003 (the recurrence),
    # 0.0001 (the latent layer, whose output is small beside the residual it is added to), and
    # 0.018 for whole models, in which every layer's roundings travel on
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    return {"rel": {"model": 2e-2, "attention": 4e-3, "mlp": 5e-3, "head": 5e-3, "experts": 3e-3,
                    "delta": 1e-2, "latent": 1e-3}[case["kind"]]}


# ------------------------------------------------------------------------ the same in 64 bits

def _w(name, shape, seed, dtype=torch.bfloat16):
    return _matrix(name, shape, seed, dtype).double()


def _unit_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, base, dims, halves):
    """``x [T, H, D]``: the first ``dims`` coordinates of every head turned."""
    half = dims // 2
    freq = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    angle = positions.double()[:, None] * freq
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    out = x.clone()
    if halves:
        u, v = x[..., :half], x[..., half:dims]
        out[..., :half], out[..., half:dims] = u * cos - v * sin, v * cos + u * sin
    else:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        out[..., 0:dims:2], out[..., 1:dims:2] = u * cos - v * sin, v * cos + u * sin
    return out


def _attend(q, k, v, first, scale, window=None):
    """Queries at positions ``first``...; ``[T, H, D]`` each, keys from position 0."""
    out = torch.empty((*q.shape[:2], v.shape[2]), dtype=q.dtype, device=q.device)
    place = torch.arange(first, first + q.shape[0], device=q.device)[:, None]
    key = torch.arange(k.shape[0], device=q.device)[None]
    hidden = key > place
    if window:
        hidden = hidden | (place - key >= window)
    for head in range(q.shape[1]):
        scores = (q[:, head] @ k[:, head].T) * scale
        out[:, head] = torch.softmax(scores.masked_fill(hidden, -math.inf), -1) @ v[:, head]
    return out


def _llama_attention(x, new, layer, shape, seed):
    """Attention rows of the last ``new`` of a request's rows ``x``."""
    h, heads, d = shape["hidden_size"], shape["num_attention_heads"], shape["head_dim"]
    prefix = f"model.layers.{layer}.self_attn"
    q, k, v = ((part @ _w(f"{prefix}.{name}_proj.weight", (heads * d, h), seed).T)
               .reshape(-1, heads, d) for name, part in (("q", x[-new:]), ("k", x), ("v", x)))
    place = torch.arange(x.shape[0], device=x.device)
    q = _rotate(q, place[-new:], shape["rope_theta"], d, True)
    k = _rotate(k, place, shape["rope_theta"], d, True)
    out = _attend(q, k, v, x.shape[0] - new, d ** -0.5)
    return out.reshape(new, heads * d) @ _w(f"{prefix}.o_proj.weight", (h, heads * d), seed).T


def _llama_mlp(x, layer, shape, seed, dtype=torch.bfloat16):
    h, i = shape["hidden_size"], shape["intermediate_size"]
    prefix = f"model.layers.{layer}.mlp"
    gate = x @ _w(f"{prefix}.gate_proj.weight", (i, h), seed, dtype).T
    up = x @ _w(f"{prefix}.up_proj.weight", (i, h), seed, dtype).T
    return (torch.nn.functional.silu(gate) * up) \
        @ _w(f"{prefix}.down_proj.weight", (h, i), seed, dtype).T


def _exact_model(case, seed):
    shape = SHAPES[case["shape"]]
    h, eps = shape["hidden_size"], shape["rms_norm_eps"]
    lengths = _lengths(case)
    table = _w("model.embed_tokens.weight", (VOCAB, h), seed)
    rows = [table[torch.tensor(_tokens(request, cached + new, seed), device=DEVICE)]
            for request, (cached, new) in enumerate(lengths)]
    counts = [row.shape[0] for row in rows]
    x = torch.cat(rows)
    for layer in range(case["layers"]):
        weight = [_vector(f"model.layers.{layer}.{name}.weight", (h,), seed).double()
                  for name in ("input_layernorm", "post_attention_layernorm")]
        normed = _unit_rms(x, eps) * weight[0]
        x = x + torch.cat([_llama_attention(part, part.shape[0], layer, shape, seed)
                           for part in normed.split(counts)])
        x = x + _llama_mlp(_unit_rms(x, eps) * weight[1], layer, shape, seed)
    last = torch.stack([part[-1] for part in x.split(counts)])
    last = _unit_rms(last, eps) * _vector("model.norm.weight", (h,), seed).double()
    return last @ _w("lm_head.weight", (VOCAB, h), seed).T


def _filter(x, taps):
    """``x [T, C]``, ``taps [C, n]``: a causal filter, the last tap on the token itself."""
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros((n - 1, x.shape[1])), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(n))


def _medolorn_input(x, seed):
    return x + _filter(x, _vector("l0.canon1", (MEDOLORN_WIDTH, CANON_TAPS), seed).double())


def _exact_experts(x, seed):
    h, ff, e, top = MEDOLORN_WIDTH, EXPERTS["ff"], EXPERTS["experts"], EXPERTS["top"]
    scores = torch.sigmoid(x @ _w("l0.mlp.router", (e, h), seed).T)
    chosen = torch.sort(scores, dim=1, descending=True, stable=True)[1][:, :top]
    weights = torch.gather(scores, 1, chosen)
    weights = weights / (weights.sum(1, keepdim=True) + 1e-20) * EXPERTS["scale"]
    out = torch.zeros_like(x)
    for expert in range(e):
        token, place = torch.nonzero(chosen == expert, as_tuple=True)
        if token.numel():
            gate, up, down = (_w(f"l0.mlp.e{expert}.{name}", shape, seed) for name, shape in
                              (("gate", (ff, h)), ("up", (ff, h)), ("down", (h, ff))))
            rows = x[token]
            act = torch.nn.functional.silu(rows @ gate.T) * (rows @ up.T)
            out.index_add_(0, token, (act @ down.T) * weights[token, place][:, None])
    return out


def _exact_delta(x, seed):
    h, heads, kv, d, vd = (MEDOLORN_WIDTH, DELTA["heads"], DELTA["kv_heads"], DELTA["dim"],
                           DELTA["vdim"])
    x = _medolorn_input(x, seed)

    def part(name, count, size):
        rows = x @ _w(f"l0.mix.{name}", (count * size, h), seed).T
        taps = _vector(f"l0.mix.{name}.conv", (count * size, DELTA["conv"]), seed).double()
        return torch.nn.functional.silu(_filter(rows, taps)).reshape(-1, count, size)
    q, k, v = part("q", kv, d), part("k", kv, d), part("v", heads, vd)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = (t.repeat_interleave(heads // kv, dim=1) for t in (q, k))
    beta = torch.sigmoid(x @ _w("l0.mix.b", (heads, h), seed).T)
    rate = torch.exp(_vector("l0.mix.A_log", (heads,), seed).double())
    step = torch.nn.functional.softplus(x @ _w("l0.mix.a", (heads, h), seed).T
                                        + _vector("l0.mix.dt_bias", (heads,), seed).double())
    decay = torch.exp(-rate * step)
    state = torch.zeros((heads, d, vd), dtype=torch.float64, device=DEVICE)
    out = torch.empty_like(v)
    for t in range(x.shape[0]):
        state = state * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", state, k[t]))
        state = state + k[t, :, :, None] * u[:, None]
        out[t] = torch.einsum("hdv,hd->hv", state, q[t])
    out = _unit_rms(out, MEDOLORN_EPS) * _vector("l0.mix.norm", (vd,), seed).double()
    gate = torch.nn.functional.silu(x @ _w("l0.mix.g", (heads * vd, h), seed).T)
    return (out.reshape(-1, heads * vd) * gate) @ _w("l0.mix.o", (h, heads * vd), seed).T


def _exact_latent(x, new, seed):
    h, heads, d, rot = MEDOLORN_WIDTH, LATENT["heads"], LATENT["dim"], LATENT["rot_dim"]
    vd, rank, qr = LATENT["vdim"], LATENT["kv_rank"], LATENT["q_rank"]
    total = x.shape[0]
    x = _medolorn_input(x, seed)
    last = x[-new:]
    place = torch.arange(total, device=DEVICE)
    latent = _unit_rms(last @ _w("l0.mix.dq", (qr, h), seed).T, MEDOLORN_EPS) \
        * _vector("l0.mix.dq.norm", (qr,), seed).double()
    q = (latent @ _w("l0.mix.uq", (heads * (d + rot), qr), seed).T).reshape(new, heads, d + rot)
    down = x @ _w("l0.mix.dkv", (rank + rot, h), seed).T
    c = _unit_rms(down[:, :rank], MEDOLORN_EPS) \
        * _vector("l0.mix.dkv.norm", (rank,), seed).double()
    shared = _rotate(down[:, rank:].reshape(total, 1, rot), place, LATENT["rot_base"],
                     LATENT["rot_dims"], False)
    turned = _rotate(q[..., d:], place[-new:], LATENT["rot_base"], LATENT["rot_dims"], False)
    k = (c @ _w("l0.mix.uk", (heads * d, rank), seed).T).reshape(total, heads, d)
    v = (c @ _w("l0.mix.uv", (heads * vd, rank), seed).T).reshape(total, heads, vd)
    out = _attend(torch.cat([q[..., :d], turned], -1),
                  torch.cat([k, shared.expand(-1, heads, -1)], -1), v, total - new,
                  LATENT["scale"], LATENT["window"])
    gate = torch.sigmoid(last @ _w("l0.mix.g", (heads * vd, h), seed).T)
    return (out.reshape(new, heads * vd) * gate) @ _w("l0.mix.o", (h, heads * vd), seed).T


def exact(case, seed):
    with torch.no_grad():
        return _exact(case, seed)


def _exact(case, seed):
    kind, dtype = case["kind"], _dtype(case)
    if kind == "model":
        return _exact_model(case, seed)
    shape = SHAPES.get(case.get("shape"), {})
    width = shape.get("hidden_size", MEDOLORN_WIDTH)
    lengths = _lengths(case)
    n = sum(new for _, new in lengths)
    before = torch.randn((n, width), generator=_generator(seed, "residual"),
                         device=DEVICE).double()
    if kind == "head":
        normed = _unit_rms(before, shape["rms_norm_eps"]) \
            * _vector("model.norm.weight", (width,), seed).double()
        return normed.flip(0) @ _w("lm_head.weight", (VOCAB, width), seed).T
    rows = [_rows(request, cached + new, width, seed, dtype).double()
            for request, (cached, new) in enumerate(lengths)]
    if kind == "mlp":
        added = _llama_mlp(torch.cat(rows), 0, shape, seed, dtype)
    elif kind == "experts":
        added = _exact_experts(torch.cat(rows), seed)
    elif kind == "delta":
        added = torch.cat([_exact_delta(part, seed) for part in rows])
    elif kind == "latent":
        added = torch.cat([_exact_latent(part, new, seed)
                           for part, (_, new) in zip(rows, lengths)])
    else:
        added = torch.cat([_llama_attention(part, new, 0, shape, seed)
                           for part, (_, new) in zip(rows, lengths)])
    out = {"residual": before + added}
    if kind in ("attention", "latent"):
        out.update(keys=None, values=None)
    if kind == "delta":
        out["state"] = None
    return out
