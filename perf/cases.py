"""Measured cases: what a program that serves models through this framework has it do.

Each case is one call through a public entry point: a step of a whole model (``ModelRunner.step``), a
layer (``blocks[i].forward``), a mixer or a feed-forward (``build_part(..).forward``), or the selection of
the next tokens (``Sampler.sample``).  Sizes are those of the benchmark's ``0.5b`` and ``1.5b`` models and
of the designs it measures at those sizes.  ``exact`` states every one of them in 64 bits.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from einf_b200.config import EngineConfig, config_from_dict
from einf_b200.config.specs import PartSpec
from einf_b200.engine import ModelRunner
from einf_b200 import ops
from einf_b200.cache.control import SamplingParams
from einf_b200.engine.batch import StepInputBuilder
from einf_b200.parts.base import CacheView, Runtime, build_part
from einf_b200.sampling import Sampler

PAGE = 16
EPS = 1e-6
DEVICE = "cuda:0"
F64 = torch.float64
SIZES = {
    "0.5b": dict(width=896, ff=4864, heads=14, kv_heads=2, size=64, vocab=151936, layers=24),
    "1.5b": dict(width=1536, ff=8960, heads=12, kv_heads=2, size=128, vocab=151936, layers=28),
}


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call of a chat with one user: one token of the whole model, bound by latency and launches
        dict(name="decode-1", kind="qwen_step", model="0.5b", requests=1, context=1024),
        # the benchmark's headline: eight users at contexts of 4,096
        dict(name="decode-8", kind="qwen_step", model="0.5b", requests=8, context=4096),
        # a layer of the larger model in a serving step: a long prompt, a short one, and a user who decodes beside them
        dict(name="layer-prompts", kind="qwen_layer", model="1.5b", dtype="bfloat16", prompts="4096,700,1", cached=0),
        # the 32-bit path, by which users check a model (`--dtype float32`, `--compare-reference`)
        dict(name="layer-32bit", kind="qwen_layer", model="0.5b", dtype="float32", prompts="512,33", cached=0),
        # linear attention over prompts
        dict(name="lightning-prompts", kind="lightning", model="0.5b", prompts="4096,1000", continued=False),
        # a state-space layer over a portion of a prompt that goes on from earlier portions
        dict(name="mamba2-portion", kind="mamba2", model="1.5b", prompts="2048", continued=True),
        # a matrix memory over prompts
        dict(name="memory-prompts", kind="memory", model="1.5b", prompts="2048,500"),
        # a whole layer with score-mixing attention beside a gated recurrence, one prompt
        dict(name="mixed-layer-prompt", kind="kanavik_layer", model="0.5b", prompts="2048"),
        # a serving step of that design: 64 users, one token each
        dict(name="mixed-decode-64", kind="kanavik_step", model="0.5b", layers=4, requests=64, context=2048),
        # a routed feed-forward over the tokens of a prompt, two of eight experts
        dict(name="routed-prompt", kind="routed", model="1.5b", experts=8, top=2, tokens=2048),
        # latent attention with rows of 512 + 64 over a prompt
        dict(name="latent-prompt", kind="latent", model="1.5b", rank=512, rot=64, prompts="2048", window=0),
        # the next tokens of eight users who sample with top-k and top-p
        dict(name="sample-8", kind="sample", rows=8, vocab=151936, top_k=50, top_p=0.9, temperature=0.8),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _prompts(rng, most):
    """One to four portions, odd lengths among them, together between 192 and `most` tokens."""
    total = _log(rng, 192, most)
    cuts = sorted(rng.randrange(1, total) for _ in range(rng.choice((0, 0, 1, 2, 3))))
    lengths = [b - a for a, b in zip([0] + cuts, cuts + [total])]
    return ",".join(str(n) for n in lengths if n > 0)


def draw(rng):
    kind = rng.choice(("qwen_step", "qwen_layer", "qwen_layer32", "lightning", "mamba2", "memory", "kanavik_layer",
                       "kanavik_step", "routed", "latent", "sample"))
    model = rng.choice(("0.5b", "1.5b"))
    if kind == "qwen_step":
        return dict(kind=kind, model="0.5b", requests=_log(rng, 1, 8), context=_log(rng, 64, 4096))
    if kind == "qwen_layer":
        return dict(kind=kind, model=model, dtype="bfloat16", prompts=_prompts(rng, 4096),
                    cached=rng.choice((0, _log(rng, 16, 2048))))
    if kind == "qwen_layer32":
        return dict(kind="qwen_layer", model="0.5b", dtype="float32", prompts=_prompts(rng, 512),
                    cached=rng.choice((0, _log(rng, 16, 512))))
    if kind in ("lightning", "mamba2"):
        return dict(kind=kind, model=model, prompts=_prompts(rng, 4096 if kind == "lightning" else 2048),
                    continued=rng.random() < 0.5)
    if kind == "memory":
        return dict(kind=kind, model=model, prompts=_prompts(rng, 2048))
    if kind == "kanavik_layer":
        return dict(kind=kind, model="0.5b", prompts=_prompts(rng, 2048))
    if kind == "kanavik_step":
        return dict(kind=kind, model="0.5b", layers=rng.choice((2, 3, 4)), requests=_log(rng, 1, 64),
                    context=_log(rng, 64, 2048))
    if kind == "routed":
        return dict(kind=kind, model=model, experts=rng.choice((4, 8)), top=rng.choice((1, 2)), tokens=_log(rng, 96, 2048))
    if kind == "latent":
        rank, rot = rng.choice(((512, 64), (256, 64), (192, 64), (448, 64)))
        return dict(kind=kind, model=model, rank=rank, rot=rot, prompts=_prompts(rng, 2048),
                    window=rng.choice((0, _log(rng, 128, 1024))))
    return dict(kind=kind, rows=_log(rng, 1, 64), vocab=rng.choice((32000, 151936, 152064)),
                top_k=rng.choice((0, 20, 50)), top_p=rng.choice((0.8, 0.9, 0.95)), temperature=rng.choice((0.6, 0.8, 1.0)))


# --------------------------------------------------------------------------- values from a seed
class _Draw:
    """Tensors in one fixed order from one generator on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(1000003 * int(seed) + 17)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return (torch.randn(shape, generator=self.g, device=DEVICE) * std + mean).to(dtype)

    def matrix(self, *shape):
        return self.normal(*shape, std=shape[-1] ** -0.5)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(shape, generator=self.g, device=DEVICE) * (high - low) + low

    def ints(self, high, count):
        return torch.randint(0, high, (count,), generator=self.g, device=DEVICE)


def _lengths(case):
    return [int(n) for n in case["prompts"].split(",")]


def _split(values, lengths):
    return torch.split(values, lengths)


def _bits64(weights):
    return {name: t.to(F64) for name, t in weights.items()}


# --------------------------------------------------------------------------- a step's inputs for a part or a layer
def _pages(requests, contexts, window, seed, capacity=None):
    """Block tables over a pool in no order: the pages that a request whose sequence is `contexts[i]` long and whose
    portion starts at `requests[i][0]` reads or writes; -1 where a window has passed."""
    need = []
    for (start, _), end in zip(requests, contexts):
        first = max(0, start - window + 1) // PAGE if window else 0
        need.append((first, -(-end // PAGE)))
    total = sum(b - a for a, b in need)
    order = torch.randperm(total, generator=torch.Generator().manual_seed(int(seed))).tolist()
    tables, at = [], 0
    for first, last in need:
        tables.append([-1] * first + order[at:at + last - first])
        at += last - first
    return tables, total


def _context(lengths, starts, tokens, seed, paged, window=0, vocab=151936):
    ends = [s + n for s, n in zip(starts, lengths)]
    tables, total = _pages(list(zip(starts, lengths)), ends, window, seed) if paged else ([[]] * len(lengths), 0)
    builder = StepInputBuilder(
        torch.device(DEVICE), PAGE, [total] if paged else [], [window or None] if paged else [], vocab,
        max(1, -(-max(ends) // PAGE)), max_tokens=sum(lengths), max_requests=len(lengths))
    rows = _split(tokens.cpu(), lengths)
    requests = [SimpleNamespace(request_id=str(i), input_token_ids=rows[i].tolist(), start_position=starts[i],
                                block_tables=[tables[i]] if paged else [], state_slot=i, need_sample=False)
                for i in range(len(lengths))]
    ctx, _ = builder.build(requests)
    return ctx, tables, total, builder


def _fill(pages, table, rows):
    """Put rows [length, heads, size] of one request's earlier tokens into its pages [pages, heads, PAGE, size]."""
    length = rows.shape[0]
    places = torch.tensor(table, device=rows.device)
    at = torch.arange(length, device=rows.device)
    page = places[at // PAGE]
    keep = page >= 0
    pages[page[keep], :, (at % PAGE)[keep]] = rows[keep]


def _runtime(dtype="bfloat16"):
    return Runtime(getattr(torch, dtype), torch.device(DEVICE))


def _libraries(category, spec, runtime):
    from einf_b200.parts.base import part_class, walk_part_specs
    names = []
    for nested_category, nested in walk_part_specs(category, spec):
        names += part_class(nested_category, nested.kind).kernel_libraries(nested, runtime)
    ops.ensure_built(tuple(dict.fromkeys(names)))


def _build(category, spec, weights, runtime):
    _libraries(category, spec, runtime)
    return build_part(category, spec, weights, runtime)


# --------------------------------------------------------------------------- statements in 64 bits
def _rms(x, weight, eps=EPS):
    y = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu(z):
    return z * torch.sigmoid(z)


def _rope(x, positions, theta, interleaved=False, table=None, amplitude=1.0):
    """x [T, heads, dims]."""
    dims = x.shape[-1]
    if table is None:
        table = theta ** (-torch.arange(0, dims, 2, device=x.device, dtype=F64) / dims)
    angle = positions.to(F64)[:, None, None] * table
    cos, sin = amplitude * torch.cos(angle), amplitude * torch.sin(angle)
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * cos - v * sin, v * cos + u * sin], dim=-1).flatten(-2)
    u, v = x[..., :dims // 2], x[..., dims // 2:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], dim=-1)


def _visible(start, length, end, window, device):
    i = torch.arange(start, start + length, device=device)[:, None]
    j = torch.arange(end, device=device)[None, :]
    mask = j <= i
    return mask & (i - j < window) if window else mask


def _conv(rows, before, weight, bias=None):
    """Causal convolution per channel: rows [T, C], before [taps - 1, C], weight [C, taps]; and the rows behind it."""
    taps = weight.shape[1]
    padded = torch.cat([before, rows])
    out = sum(padded[j:j + rows.shape[0]] * weight[:, j] for j in range(taps))
    return (out if bias is None else out + bias), padded[rows.shape[0]:]


# --------------------------------------------------------------------------- Qwen2: layers and whole steps
def _qwen_config(case, layers):
    s = SIZES[case["model"]]
    return dict(architectures=["Qwen2ForCausalLM"], vocab_size=s["vocab"] if case["kind"] == "qwen_step" else 4096,
                hidden_size=s["width"], intermediate_size=s["ff"], num_hidden_layers=layers,
                num_attention_heads=s["heads"], num_key_value_heads=s["kv_heads"], rms_norm_eps=EPS, hidden_act="silu",
                rope_theta=1000000.0, max_position_embeddings=32768, tie_word_embeddings=True, bos_token_id=151643,
                eos_token_id=151643)


def _qwen_weights(d, cfg):
    h, ff, heads, kv = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    size = h // heads
    w = {"model.embed_tokens.weight": d.normal(cfg["vocab_size"], h), "model.norm.weight": d.normal(h, std=0.05, mean=1.0)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, rows in (("q", heads * size), ("k", kv * size), ("v", kv * size)):
            w[p + f"self_attn.{name}_proj.weight"] = d.matrix(rows, h)
            w[p + f"self_attn.{name}_proj.bias"] = d.normal(rows, std=0.1)
        w[p + "self_attn.o_proj.weight"] = d.matrix(h, heads * size)
        w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"] = d.matrix(ff, h), d.matrix(ff, h)
        w[p + "mlp.down_proj.weight"] = d.matrix(h, ff)
        for norm in ("input_layernorm", "post_attention_layernorm"):
            w[p + norm + ".weight"] = d.normal(h, std=0.05, mean=1.0)
    return w


def _qwen_layer_exact(x, positions, starts, lengths, w, p, cfg, earlier):
    """One layer over packed portions; earlier(request) -> keys, values of the tokens before a portion."""
    heads, kv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    size = cfg["hidden_size"] // heads
    h = _rms(x, w[p + "input_layernorm.weight"])
    q, k, v = (h @ w[p + f"self_attn.{n}_proj.weight"].T + w[p + f"self_attn.{n}_proj.bias"] for n in "qkv")
    q = _rope(q.view(-1, heads, size), positions, cfg["rope_theta"])
    k = _rope(k.view(-1, kv, size), positions, cfg["rope_theta"])
    v = v.view(-1, kv, size)
    out = []
    for r, (qr, kr, vr) in enumerate(zip(_split(q, lengths), _split(k, lengths), _split(v, lengths))):
        if starts[r]:
            before_k, before_v = earlier(r)
            kr, vr = torch.cat([before_k, kr]), torch.cat([before_v, vr])
        mask = _visible(starts[r], lengths[r], starts[r] + lengths[r], 0, x.device)
        mixed = []
        for a in range(heads):
            scores = (qr[:, a] @ kr[:, a // (heads // kv)].T) * size ** -0.5
            mixed.append(torch.softmax(scores.masked_fill(~mask, -math.inf), -1) @ vr[:, a // (heads // kv)])
        out.append(torch.cat(mixed, dim=1))
    x = x + torch.cat(out) @ w[p + "self_attn.o_proj.weight"].T
    h = _rms(x, w[p + "post_attention_layernorm.weight"])
    ff = _silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
    return x, ff @ w[p + "mlp.down_proj.weight"].T, k, v


def _earlier(d, length, kv, size, dtype):
    return d.normal(length, kv, size, dtype=dtype), d.normal(length, kv, size, dtype=dtype)


def _qwen_layer_values(case, seed):
    d, cfg = _Draw(seed), _qwen_config(case, 1)
    dtype = getattr(torch, case["dtype"])
    lengths, cached = _lengths(case), case["cached"]
    size = cfg["hidden_size"] // cfg["num_attention_heads"]
    weights = _qwen_weights(d, cfg)
    x = d.normal(sum(lengths), cfg["hidden_size"], dtype=torch.float32)
    tokens = d.ints(4096, sum(lengths))
    rows = [_earlier(d, cached, cfg["num_key_value_heads"], size, dtype) for _ in lengths] if cached else None
    return cfg, weights, x, tokens, lengths, rows


def _prepare_qwen_layer(case, seed):
    cfg, weights, x, tokens, lengths, rows = _qwen_layer_values(case, seed)
    cached = case["cached"]
    total = sum(-(-(n + cached) // PAGE) for n in lengths)
    runner = ModelRunner(config_from_dict(cfg), weights, EngineConfig(
        dtype=case["dtype"], block_len=PAGE, num_blocks=total, max_batch_len=sum(lengths),
        max_prefill_chunk_len=max(lengths), max_requests=len(lengths)))
    tables, _ = _pages([(cached, n) for n in lengths], [cached + n for n in lengths], 0, seed)
    split = _split(tokens.cpu(), lengths)
    view = runner.storage.views[0]
    if cached:
        for table, (k, v) in zip(tables, rows):
            _fill(view.k, table, k)
            _fill(view.v, table, v)
    requests = [SimpleNamespace(request_id=str(i), input_token_ids=split[i].tolist(), start_position=cached,
                                block_tables=[tables[i]], state_slot=-1, need_sample=False) for i in range(len(lengths))]
    ctx, _ = runner.inputs.build(requests)
    return dict(run=_run_qwen_layer, block=runner.model.blocks[0], ctx=ctx, view=view, x=x, keep=runner,
                residual=torch.empty_like(x))


def _run_qwen_layer(s):
    s["residual"].copy_(s["x"])         # the step's embedding kernel writes the stream anew
    pending = s["block"].forward(s["residual"], None, s["ctx"], s["view"])
    return {"stream": s["residual"], "pending": pending}


def _exact_qwen_layer(case, seed):
    cfg, weights, x, tokens, lengths, rows = _qwen_layer_values(case, seed)
    cached = case["cached"]
    starts = [cached] * len(lengths)
    positions = torch.cat([torch.arange(cached, cached + n, device=DEVICE) for n in lengths])
    x, pending, _, _ = _qwen_layer_exact(x.to(F64), positions, starts, lengths, _bits64(weights), "model.layers.0.", cfg,
                                         lambda r: (rows[r][0].to(F64), rows[r][1].to(F64)))
    return {"stream": x, "pending": pending}


def _qwen_step_values(case, seed):
    d, cfg = _Draw(seed), _qwen_config(case, SIZES[case["model"]]["layers"])
    weights = _qwen_weights(d, cfg)
    tokens = d.ints(cfg["vocab_size"], case["requests"])
    size = cfg["hidden_size"] // cfg["num_attention_heads"]

    def rows(layer, request):
        g = _Draw(seed * 7919 + layer * 101 + request + 1)
        return _earlier(g, case["context"], cfg["num_key_value_heads"], size, torch.bfloat16)
    return cfg, weights, tokens, rows


def _prepare_qwen_step(case, seed):
    cfg, weights, tokens, rows = _qwen_step_values(case, seed)
    count, context = case["requests"], case["context"]
    tables, total = _pages([(context, 1)] * count, [context + 1] * count, 0, seed)
    runner = ModelRunner(config_from_dict(cfg), weights, EngineConfig(
        dtype="bfloat16", block_len=PAGE, num_blocks=total, max_batch_len=256, max_prefill_chunk_len=256,
        max_requests=8, max_sequence_len=context + 64))
    for layer, view in enumerate(runner.storage.views):
        for r in range(count):
            k, v = rows(layer, r)
            _fill(view.k, tables[r], k)
            _fill(view.v, tables[r], v)
    requests = [SimpleNamespace(request_id=str(i), input_token_ids=[t], start_position=context, block_tables=[tables[i]],
                                state_slot=-1, need_sample=True) for i, t in enumerate(tokens.tolist())]
    return dict(run=_run_step, runner=runner, requests=requests)


def _run_step(s):
    return {"logits": s["runner"].step(s["requests"]).logits}


def _exact_qwen_step(case, seed):
    cfg, weights, tokens, rows = _qwen_step_values(case, seed)
    count, context = case["requests"], case["context"]
    w = _bits64(weights)
    x = w["model.embed_tokens.weight"][tokens]
    positions = torch.full((count,), context, device=DEVICE)
    for layer in range(cfg["num_hidden_layers"]):
        x, pending, _, _ = _qwen_layer_exact(x, positions, [context] * count, [1] * count, w, f"model.layers.{layer}.", cfg,
                                             lambda r: tuple(t.to(F64) for t in rows(layer, r)))
        x = x + pending
    return {"logits": _rms(x, w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T}


# --------------------------------------------------------------------------- recurrent mixers
def _recurrent_state(case, floats, count, d, std):
    """The state rows before the call: of requests that start here, cleared by the step; else of earlier portions."""
    return d.normal(count, floats, std=std if case.get("continued") else 0.0, dtype=torch.float32)


def _prepare_recurrent(case, seed, spec, weights, x, state):
    runtime = _runtime()
    part = _build("mixer", spec, weights, runtime)
    lengths = _lengths(case)
    starts = [1024 if case.get("continued") else 0] * len(lengths)
    ctx, _, _, builder = _context(lengths, starts, torch.zeros(sum(lengths), dtype=torch.int64), seed, paged=False)
    need = part.cache_need().shape[0]
    if state is None:
        state = torch.zeros((len(lengths), need), dtype=torch.float32, device=DEVICE)
    assert state.shape[1] == need
    return dict(run=_run_recurrent, part=part, ctx=ctx, x=x, state=state, view=CacheView(state=state), keep=builder)


def _run_recurrent(s):
    ctx = s["ctx"]
    ops.zero_fresh_state(s["state"], ctx.state_slots, ctx.q_start, ctx.positions)     # as every step begins
    return {"out": s["part"].forward(s["x"], ctx, s["view"]), "state": s["state"]}


def _lightning_values(case, seed):
    d, s, lengths = _Draw(seed), SIZES[case["model"]], _lengths(case)
    h, heads, dim = s["width"], s["heads"], s["size"]
    w = {n + "_proj.weight": d.matrix(heads * dim, h) for n in "qkvg"}
    w["o_proj.weight"] = d.matrix(h, heads * dim)
    w["norm.weight"] = d.normal(heads * dim, std=0.1, mean=1.0)
    decay = [1.0 - 2.0 ** -(3 + 6 * a / heads) for a in range(heads)]
    x = d.normal(sum(lengths), h)
    state = _recurrent_state(case, heads * dim * dim, len(lengths), d, 1.0)
    return w, decay, x, state, lengths, heads, dim, h


def _prepare_lightning(case, seed):
    w, decay, x, state, lengths, heads, dim, h = _lightning_values(case, seed)
    spec = PartSpec("lightning", {"hidden_size": h, "num_heads": heads, "head_size": dim, "value_head_size": dim,
                                  "decay": tuple(decay), "eps": EPS})
    return _prepare_recurrent(case, seed, spec, w, x, state)


def _exact_lightning(case, seed):
    w, decay, x, state, lengths, heads, dim, h = _lightning_values(case, seed)
    w, x = _bits64(w), x.to(F64)
    q, k, v = (_silu(x @ w[n + "_proj.weight"].T).view(-1, heads, dim) for n in "qkv")
    keep = torch.tensor(decay, device=DEVICE).to(F64)[:, None, None]
    states, rows = [], []
    for r, (qr, kr, vr) in enumerate(zip(*(_split(t, lengths) for t in (q, k, v)))):
        S = state[r].to(F64).view(heads, dim, dim)
        for t in range(lengths[r]):
            S = keep * S + kr[t][:, :, None] * vr[t][:, None, :]
            rows.append(torch.matmul(qr[t][:, None, :], S).reshape(-1))
        states.append(S.reshape(-1))
    y = _rms(torch.stack(rows), w["norm.weight"]) * torch.sigmoid(x @ w["g_proj.weight"].T)
    return {"out": y @ w["o_proj.weight"].T, "state": torch.stack(states)}


def _mamba2_values(case, seed):
    d, s, lengths = _Draw(seed), SIZES[case["model"]], _lengths(case)
    h, P, N, G, taps = s["width"], 64, 128, 1, 4
    heads = s["heads"] * s["size"] // P
    inner, channels = heads * P, heads * P + 2 * G * N
    w = {"in_proj.weight": d.matrix(inner + channels + heads, h), "conv.weight": d.normal(channels, taps, std=taps ** -0.5),
         "conv.bias": d.normal(channels, std=0.1)}
    # steps of 0.001 to 0.1 before the token's own part, rates of 1 to 16
    dt = torch.exp(d.uniform(heads, low=math.log(1e-3), high=math.log(1e-1)))
    w["dt_bias"] = torch.log(torch.expm1(dt)).to(torch.bfloat16)
    w["A_log"] = torch.log(d.uniform(heads, low=1.0, high=16.0)).to(torch.bfloat16)
    w["D"] = d.normal(heads, std=0.2, mean=1.0)
    w["norm.weight"] = d.normal(inner, std=0.1, mean=1.0)
    w["o_proj.weight"] = d.matrix(h, inner)
    x = d.normal(sum(lengths), h)
    state = torch.cat([_recurrent_state(case, heads * N * P, len(lengths), d, 0.3),
                       _recurrent_state(case, (taps - 1) * channels, len(lengths), d, 1.0)], dim=1)
    return w, x, state, lengths, h, heads, P, N, G, taps, inner, channels


def _prepare_mamba2(case, seed):
    w, x, state, lengths, h, heads, P, N, G, taps, inner, channels = _mamba2_values(case, seed)
    spec = PartSpec("mamba2", {"hidden_size": h, "num_heads": heads, "value_head_size": P, "state_size": N,
                               "num_groups": G, "conv_taps": taps, "norm_groups": 1, "eps": EPS})
    return _prepare_recurrent(case, seed, spec, w, x, state)


def _exact_mamba2(case, seed):
    w, x, state, lengths, h, heads, P, N, G, taps, inner, channels = _mamba2_values(case, seed)
    w, x, state = _bits64(w), x.to(F64), state.to(F64)
    proj = x @ w["in_proj.weight"].T
    z, xbc, raw = proj[:, :inner], proj[:, inner:inner + channels], proj[:, inner + channels:]
    dt = torch.nn.functional.softplus(raw + w["dt_bias"])
    keep = torch.exp(-torch.exp(w["A_log"]) * dt)
    rows, states = [], []
    for r, (part, dtr, kr) in enumerate(zip(*(_split(t, lengths) for t in (xbc, dt, keep)))):
        conv, behind = _conv(part, state[r, heads * N * P:].view(taps - 1, channels), w["conv.weight"], w["conv.bias"])
        conv = _silu(conv)
        xs, B, C = conv[:, :inner].view(-1, heads, P), conv[:, inner:inner + N], conv[:, inner + N:]
        S = state[r, :heads * N * P].view(heads, N, P)
        for t in range(lengths[r]):
            S = kr[t][:, None, None] * S + B[t][None, :, None] * (dtr[t][:, None] * xs[t])[:, None, :]
            rows.append((torch.matmul(C[t], S) + w["D"][:, None] * xs[t]).reshape(-1))
        states.append(torch.cat([S.reshape(-1), behind.reshape(-1)]))
    y = _rms(torch.stack(rows) * _silu(z), w["norm.weight"])
    return {"out": y @ w["o_proj.weight"].T, "state": torch.stack(states)}


def _memory_values(case, seed):
    d, s, lengths = _Draw(seed), SIZES[case["model"]], _lengths(case)
    h, heads, dim = s["width"], s["heads"] // 2, s["size"]
    vdim = h // heads
    w = {"q_proj.weight": d.matrix(heads * dim, h), "k_proj.weight": d.matrix(heads * dim, h),
         "v_proj.weight": d.matrix(heads * vdim, h), "g_proj.weight": d.matrix(heads * vdim, h),
         "i_proj.weight": d.matrix(heads, h), "i_proj.bias": d.normal(heads, std=0.3),
         "f_proj.weight": d.matrix(heads, h), "f_proj.bias": d.normal(heads, std=0.5, mean=4.0),
         "norm.weight": d.normal(heads * vdim, std=0.1, mean=1.0), "o_proj.weight": d.matrix(h, heads * vdim)}
    return w, d.normal(sum(lengths), h), lengths, h, heads, dim, vdim


def _prepare_memory(case, seed):
    w, x, lengths, h, heads, dim, vdim = _memory_values(case, seed)
    spec = PartSpec("matrix_memory", {"hidden_size": h, "num_heads": heads, "head_size": dim, "value_head_size": vdim,
                                      "eps": EPS, "gate_cap": 15.0, "denominator_eps": 1e-6})
    return _prepare_recurrent(case, seed, spec, w, x, None)


def _exact_memory(case, seed):
    w, x, lengths, h, heads, dim, vdim = _memory_values(case, seed)
    w, x = _bits64(w), x.to(F64)
    q = (x @ w["q_proj.weight"].T).view(-1, heads, dim) * dim ** -0.5
    k = (x @ w["k_proj.weight"].T).view(-1, heads, dim)
    v = (x @ w["v_proj.weight"].T).view(-1, heads, vdim)
    log_in = 15.0 * torch.tanh((x @ w["i_proj.weight"].T + w["i_proj.bias"]) / 15.0)
    log_keep = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w["f_proj.weight"].T + w["f_proj.bias"]) / 15.0))
    wide = torch.cat([v, torch.ones_like(v[:, :, :1])], dim=2)      # the normaliser as one more column
    rows, floors = [], []
    for qr, kr, vr, li, lk in zip(*(_split(t, lengths) for t in (q, k, wide, log_in, log_keep))):
        S = torch.zeros(heads, dim, vdim + 1, dtype=F64, device=DEVICE)
        top = torch.zeros(heads, dtype=F64, device=DEVICE)
        for t in range(qr.shape[0]):
            new = torch.maximum(lk[t] + top, li[t])
            S = torch.exp(lk[t] + top - new)[:, None, None] * S \
                + (torch.exp(li[t] - new)[:, None] * kr[t])[:, :, None] * vr[t][:, None, :]
            rows.append(torch.matmul(qr[t][:, None, :], S)[:, 0])
            top = new
            floors.append(new)
    y, top = torch.stack(rows), torch.stack(floors)
    below = torch.maximum(y[:, :, -1].abs(), torch.exp(-top)) + 1e-6
    y = _rms(y[:, :, :-1] / below[:, :, None], None).reshape(-1, heads * vdim) * w["norm.weight"]
    return {"out": (y * torch.sigmoid(x @ w["g_proj.weight"].T)) @ w["o_proj.weight"].T, "state": None}


# --------------------------------------------------------------------------- Kanavik: a layer, and whole steps
_WINDOW, _TAPS, _SIDE, _MULT = 1024, 4, 64, 0.5


def _kanavik_config(case, layers, positions, vocab):
    s = SIZES[case["model"]]
    layer = {"type": "parallel", "mixer": {
        "left": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": s["size"], "vdim": s["size"],
                 "scale": s["size"] ** -0.5, "mask": {"size": _WINDOW}}, "left_scale": 1.0,
        "right": {"width": s["width"], "blocks": s["heads"], "conv": _TAPS}, "right_scale": 1.0},
        "mlp": {"kind": "dense", "ff": s["ff"]}}
    return {"architecture": "Kanavik", "vocab": vocab, "width": s["width"], "max_positions": positions,
            "norm": {"eps": EPS}, "residual_mult": _MULT, "canon": {"taps": _TAPS}, "token_side": {"dim": _SIDE},
            "layers": [dict(layer) for _ in range(layers)]}


def _kanavik_weights(d, cfg):
    h, layers = cfg["width"], len(cfg["layers"])
    left, right = cfg["layers"][0]["mixer"]["left"], cfg["layers"][0]["mixer"]["right"]
    heads, kv, size, blocks, ff = left["heads"], left["kv_heads"], left["dim"], right["blocks"], cfg["layers"][0]["mlp"]["ff"]
    w = {"embed": d.normal(cfg["vocab"], h), "pos": d.normal(cfg["max_positions"], h, std=0.5),
         "final.norm": d.normal(h, std=0.1, mean=1.0), "head": d.matrix(cfg["vocab"], h),
         "side.embed": d.normal(cfg["vocab"], _SIDE * layers)}
    for i in range(layers):
        p = f"l{i}."
        for n in ("norm1", "norm2", "side.norm"):
            w[p + n] = d.normal(h, std=0.1, mean=1.0)
        for n in ("canon1", "canon2", "mix.right.conv"):
            w[p + n] = d.normal(h, _TAPS, std=0.4)
        w[p + "mix.left.q"], w[p + "mix.left.o"] = d.matrix(heads * size, h), d.matrix(h, heads * size)
        w[p + "mix.left.k"], w[p + "mix.left.v"] = d.matrix(kv * size, h), d.matrix(kv * size, h)
        w[p + "mix.left.talk"] = (torch.eye(heads, device=DEVICE) + d.normal(heads, heads, std=0.3).float()).to(torch.bfloat16)
        w[p + "mix.left.sink"] = d.normal(heads)
        for n in ("y", "x"):
            w[p + f"mix.right.{n}"], w[p + f"mix.right.{n}.b"] = d.matrix(h, h), d.normal(h, std=0.3)
        w[p + "mix.right.conv.b"] = d.normal(h, std=0.3)
        for n in ("ra", "ri"):
            w[p + f"mix.right.{n}"] = d.matrix(blocks, h // blocks, h // blocks)
            w[p + f"mix.right.{n}.b"] = d.normal(blocks, h // blocks, std=0.3)
        w[p + "mix.right.lam"] = d.normal(h, std=1.5, mean=-2.0)
        w[p + "mix.right.o"] = d.matrix(h, h)
        w[p + "mlp.gate"], w[p + "mlp.up"], w[p + "mlp.down"] = d.matrix(ff, h), d.matrix(ff, h), d.matrix(h, ff)
        average = d.normal(i + 2, std=0.2, dtype=torch.float32)
        average[-1] += 1.0
        w[p + "dwa"] = average.to(torch.bfloat16)
        w[p + "side.gate"], w[p + "side.proj"] = d.matrix(_SIDE, h), d.matrix(h, _SIDE)
    return w


def _kanavik_state_floats(cfg):
    return cfg["width"] * (2 * (_TAPS - 1) + 1 + (_TAPS - 1))


def _kanavik_layer_exact(x, tokens, history, index, starts, lengths, w, cfg, earlier, state):
    """One layer over packed portions.  earlier(request) -> keys, values; state(request) -> the row of
    [first convolution | second | S | the branch's convolution]."""
    p, h = f"l{index}.", cfg["width"]
    left = cfg["layers"][0]["mixer"]["left"]
    heads, kv, size = left["heads"], left["kv_heads"], left["dim"]
    blocks = cfg["layers"][0]["mixer"]["right"]["blocks"]
    part, behind = h // blocks, (_TAPS - 1) * h
    slopes = torch.tensor([2.0 ** (-8.0 * (a + 1) / heads) for a in range(heads)], dtype=F64, device=x.device)

    def canon(values, offset, name):
        out = []
        for r, rows in enumerate(_split(values, lengths)):
            out.append(rows + _conv(rows, state(r)[offset:offset + behind].view(_TAPS - 1, h), w[p + name])[0])
        return torch.cat(out)

    n = canon(_rms(x, w[p + "norm1"]), 0, "canon1")
    q = (n @ w[p + "mix.left.q"].T).view(-1, heads, size)
    k = (n @ w[p + "mix.left.k"].T).view(-1, kv, size)
    v = (n @ w[p + "mix.left.v"].T).view(-1, kv, size)
    mixed = []
    for r, (qr, kr, vr) in enumerate(zip(*(_split(t, lengths) for t in (q, k, v)))):
        if starts[r]:
            before_k, before_v = earlier(r)
            kr, vr = torch.cat([before_k, kr]), torch.cat([before_v, vr])
        end = starts[r] + lengths[r]
        mask = _visible(starts[r], lengths[r], end, _WINDOW, x.device)
        i = torch.arange(starts[r], end, device=x.device)[:, None]
        distance = (i - torch.arange(end, device=x.device)[None, :]).to(F64)
        raw = torch.stack([(qr[:, a] @ kr[:, a // (heads // kv)].T) * size ** -0.5 - slopes[a] * distance
                           for a in range(heads)])
        rows = []
        for a in range(heads):
            scores = torch.einsum("g,gij->ij", w[p + "mix.left.talk"][a], raw).masked_fill(~mask, -math.inf)
            sink = w[p + "mix.left.sink"][a]
            top = torch.maximum(scores.max(-1, keepdim=True).values, sink)
            e = torch.exp(scores - top)
            e = e / (e.sum(-1, keepdim=True) + torch.exp(sink - top))
            rows.append(e @ vr[:, a // (heads // kv)])
        mixed.append(torch.cat(rows, dim=1))
    out = torch.cat(mixed) @ w[p + "mix.left.o"].T
    y = _gelu(n @ w[p + "mix.right.y"].T + w[p + "mix.right.y.b"])
    branch = n @ w[p + "mix.right.x"].T + w[p + "mix.right.x.b"]
    soft = torch.nn.functional.softplus(w[p + "mix.right.lam"])
    rows = []
    for r, b in enumerate(_split(branch, lengths)):
        row = state(r)
        u, _ = _conv(b, row[2 * behind + h:2 * behind + h + behind].view(_TAPS - 1, h), w[p + "mix.right.conv"],
                     w[p + "mix.right.conv.b"])
        by = u.view(-1, blocks, part)
        gate = [torch.sigmoid(torch.einsum("bop,tbp->tbo", w[p + f"mix.right.{g}"], by) + w[p + f"mix.right.{g}.b"]).reshape(-1, h)
                for g in ("ra", "ri")]
        a = torch.exp(-8.0 * gate[0] * soft)
        add = torch.sqrt(1.0 - a * a) * gate[1] * u
        S = row[2 * behind:2 * behind + h]
        for t in range(lengths[r]):
            S = a[t] * S + add[t]
            rows.append(S)
    out = out + (torch.stack(rows) * y) @ w[p + "mix.right.o"].T
    x = x + _MULT * out
    n = canon(_rms(x, w[p + "norm2"]), behind, "canon2")
    x = x + _MULT * ((_gelu(n @ w[p + "mlp.gate"].T) * (n @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T)
    g = _gelu(x @ w[p + "side.gate"].T) * w["side.embed"][tokens][:, index * _SIDE:(index + 1) * _SIDE]
    x = x + _MULT * _rms(g @ w[p + "side.proj"].T, w[p + "side.norm"])
    history.append(x)
    return sum(w[p + "dwa"][j] * history[j] for j in range(index + 2))


def _kanavik_layer_values(case, seed):
    d, lengths = _Draw(seed), _lengths(case)
    cfg = _kanavik_config(case, 1, max(lengths), 4096)
    weights = _kanavik_weights(d, cfg)
    return cfg, weights, d.normal(sum(lengths), cfg["width"], dtype=torch.float32), d.ints(4096, sum(lengths)), lengths


def _prepare_kanavik_layer(case, seed):
    cfg, weights, x, tokens, lengths = _kanavik_layer_values(case, seed)
    total = sum(-(-n // PAGE) for n in lengths)
    runner = ModelRunner(config_from_dict(cfg), weights, EngineConfig(
        dtype="bfloat16", block_len=PAGE, num_blocks=total, max_batch_len=sum(lengths), max_prefill_chunk_len=max(lengths),
        max_requests=len(lengths)))
    tables, _ = _pages([(0, n) for n in lengths], lengths, _WINDOW, seed)
    split = _split(tokens.cpu(), lengths)
    requests = [SimpleNamespace(request_id=str(i), input_token_ids=split[i].tolist(), start_position=0,
                                block_tables=[tables[i]], state_slot=i, need_sample=False) for i in range(len(lengths))]
    ctx, _ = runner.inputs.build(requests)
    view = runner.storage.views[0]
    return dict(run=_run_kanavik_layer, block=runner.model.blocks[0], ctx=ctx, view=view, x=x, keep=runner,
                residual=torch.empty_like(x))


def _run_kanavik_layer(s):
    ctx = s["ctx"]
    ops.zero_fresh_state(s["view"].state, ctx.state_slots, ctx.q_start, ctx.positions)   # as every step begins
    s["residual"].copy_(s["x"])         # the step's embedding kernel writes the stream anew
    s["block"].forward(s["residual"], None, ctx, s["view"])
    return {"stream": s["residual"]}


def _exact_kanavik_layer(case, seed):
    cfg, weights, x, tokens, lengths = _kanavik_layer_values(case, seed)
    x = x.to(F64)
    empty = torch.zeros(_kanavik_state_floats(cfg), dtype=F64, device=DEVICE)
    out = _kanavik_layer_exact(x, tokens, [x], 0, [0] * len(lengths), lengths, _bits64(weights), cfg, None, lambda r: empty)
    return {"stream": out}


def _kanavik_step_values(case, seed):
    d, s = _Draw(seed), SIZES[case["model"]]
    cfg = _kanavik_config(case, case["layers"], case["context"] + 64, s["vocab"])
    weights = _kanavik_weights(d, cfg)
    tokens = d.ints(s["vocab"], case["requests"])

    def rows(layer, request):
        g = _Draw(seed * 7919 + layer * 101 + request + 1)
        return _earlier(g, case["context"], s["kv_heads"], s["size"], torch.bfloat16)

    def state(layer, request):
        g = _Draw(seed * 7907 + layer * 103 + request + 5)
        return g.normal(_kanavik_state_floats(cfg), dtype=torch.float32)
    return cfg, weights, tokens, rows, state


def _prepare_kanavik_step(case, seed):
    cfg, weights, tokens, rows, state = _kanavik_step_values(case, seed)
    count, context = case["requests"], case["context"]
    tables, total = _pages([(context, 1)] * count, [context + 1] * count, _WINDOW, seed)
    runner = ModelRunner(config_from_dict(cfg), weights, EngineConfig(
        dtype="bfloat16", block_len=PAGE, num_blocks=max(total, -(-(context + 64) // PAGE)), max_batch_len=256,
        max_prefill_chunk_len=256, max_requests=count))
    for layer, view in enumerate(runner.storage.views):
        for r in range(count):
            k, v = rows(layer, r)
            _fill(view.k, tables[r], k)
            _fill(view.v, tables[r], v)
            view.state[r].copy_(state(layer, r))
    requests = [SimpleNamespace(request_id=str(i), input_token_ids=[t], start_position=context, block_tables=[tables[i]],
                                state_slot=i, need_sample=True) for i, t in enumerate(tokens.tolist())]
    return dict(run=_run_step, runner=runner, requests=requests)


def _exact_kanavik_step(case, seed):
    cfg, weights, tokens, rows, state = _kanavik_step_values(case, seed)
    count, context = case["requests"], case["context"]
    w = _bits64(weights)
    x = w["embed"][tokens] + w["pos"][context]
    history = [x]
    for layer in range(case["layers"]):
        x = _kanavik_layer_exact(x, tokens, history, layer, [context] * count, [1] * count, w, cfg,
                                 lambda r: tuple(t.to(F64) for t in rows(layer, r)), lambda r: state(layer, r).to(F64))
    return {"logits": _rms(x, w["final.norm"]) @ w["head"].T}


# --------------------------------------------------------------------------- a routed feed-forward
def _routed_values(case, seed):
    d, s = _Draw(seed), SIZES[case["model"]]
    h, ff, experts = s["width"], s["ff"] // case["top"], case["experts"]
    w = {"router.weight": d.normal(experts, h, std=2.0 * h ** -0.5)}
    for e in range(experts):
        w[f"experts.{e}.gate_proj.weight"], w[f"experts.{e}.up_proj.weight"] = d.matrix(ff, h), d.matrix(ff, h)
        w[f"experts.{e}.down_proj.weight"] = d.matrix(h, ff)
    return w, d.normal(case["tokens"], h), h, ff, experts


def _prepare_routed(case, seed):
    w, x, h, ff, experts = _routed_values(case, seed)
    spec = PartSpec("routed_mlp", {"hidden_size": h, "intermediate_size": ff, "num_experts": experts, "top_k": case["top"],
                                   "score": "sigmoid", "renormalise": False, "weight_on": "output"})
    part = _build("feed_forward", spec, w, _runtime())
    n = case["tokens"]
    ctx, _, _, builder = _context([n], [0], torch.zeros(n, dtype=torch.int64), seed, paged=False)
    return dict(run=_run_routed, part=part, ctx=ctx, x=x, keep=builder)


def _run_routed(s):
    return {"out": s["part"].forward(s["x"], s["ctx"])}


def _exact_routed(case, seed):
    w, x, h, ff, experts = _routed_values(case, seed)
    w, x = _bits64(w), x.to(F64)
    scores = torch.sigmoid(x @ w["router.weight"].T)
    weight, chosen = torch.topk(scores, case["top"], dim=1)
    out = torch.zeros_like(x)
    for e in range(experts):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        u = x[rows]
        y = (_silu(u @ w[f"experts.{e}.gate_proj.weight"].T) * (u @ w[f"experts.{e}.up_proj.weight"].T)) \
            @ w[f"experts.{e}.down_proj.weight"].T
        out[rows] += weight[rows, place][:, None] * y
    return {"out": out}


# --------------------------------------------------------------------------- latent attention
_YARN = {"factor": 8.0, "original": 4096.0, "fast": 32.0, "slow": 1.0}


def _latent_values(case, seed):
    d, s, lengths = _Draw(seed), SIZES[case["model"]], _lengths(case)
    h, heads, dim, rank, rot = s["width"], s["heads"], s["size"], case["rank"], case["rot"]
    w = {"q_proj.weight": d.matrix(heads * (dim + rot), h), "sink": d.normal(heads, std=0.5),
         "kv_down.weight": d.matrix(rank + rot, h), "kv_norm.weight": d.normal(rank, std=0.1, mean=1.0),
         "k_up.weight": d.matrix(heads * dim, rank), "v_up.weight": d.matrix(heads * dim, rank),
         "o_proj.weight": d.matrix(h, heads * dim)}
    return w, d.normal(sum(lengths), h), lengths, h, heads, dim, rank, rot


def _prepare_latent(case, seed):
    w, x, lengths, h, heads, dim, rank, rot = _latent_values(case, seed)
    window = case["window"] or None
    spec = PartSpec("latent_attention", {
        "hidden_size": h, "num_heads": heads, "head_size": dim, "rotary_size": rot, "value_head_size": dim, "kv_rank": rank,
        "q_rank": None, "scale": (dim + rot) ** -0.5, "eps": EPS, "window": window, "sink": True,
        "position": PartSpec("rope", {"rotary_dim": rot, "theta": 1e6, "layout": "interleaved",
                                      "scaling": dict(_YARN, kind="yarn")})})
    part = _build("mixer", spec, w, _runtime())
    tokens = torch.zeros(sum(lengths), dtype=torch.int64)
    ctx, _, total, builder = _context(lengths, [0] * len(lengths), tokens, seed, paged=True, window=case["window"])
    need = part.cache_need()
    pages = torch.zeros((total, 1, PAGE, need.head_size), dtype=torch.bfloat16, device=DEVICE)
    return dict(run=_run_latent, part=part, ctx=ctx, x=x, keep=builder,
                view=CacheView(group=0, k=pages, v=None, writes=True, page_size=PAGE))


def _run_latent(s):
    return {"out": s["part"].forward(s["x"], s["ctx"], s["view"])}


def _yarn_table(rot, theta):
    def place(turns):
        return rot * math.log(_YARN["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(theta))
    low, high = max(math.floor(place(_YARN["fast"])), 0), min(math.ceil(place(_YARN["slow"])), rot - 1)
    table = []
    for i in range(rot // 2):
        f = theta ** (-2.0 * i / rot)
        ramp = min(max((i - low) / max(high - low, 0.001), 0.0), 1.0)
        table.append(f / _YARN["factor"] * ramp + f * (1.0 - ramp))
    return torch.tensor(table, dtype=F64, device=DEVICE), 0.1 * math.log(_YARN["factor"]) + 1.0


def _exact_latent(case, seed):
    w, x, lengths, h, heads, dim, rank, rot = _latent_values(case, seed)
    w, x = _bits64(w), x.to(F64)
    positions = torch.cat([torch.arange(n, device=DEVICE) for n in lengths])
    table, amplitude = _yarn_table(rot, 1e6)
    q = (x @ w["q_proj.weight"].T).view(-1, heads, dim + rot)
    q_rot = _rope(q[..., dim:], positions, 0.0, True, table, amplitude)
    down = x @ w["kv_down.weight"].T
    latent = _rms(down[:, :rank], w["kv_norm.weight"])
    shared = _rope(down[:, None, rank:], positions, 0.0, True, table, amplitude)[:, 0]
    k = (latent @ w["k_up.weight"].T).view(-1, heads, dim)
    v = (latent @ w["v_up.weight"].T).view(-1, heads, dim)
    out = []
    for r, (qp, qr, kr, sr, vr) in enumerate(zip(*(_split(t, lengths) for t in (q[..., :dim], q_rot, k, shared, v)))):
        mask = _visible(0, lengths[r], lengths[r], case["window"], x.device)
        mixed = []
        for a in range(heads):
            scores = ((qp[:, a] @ kr[:, a].T + qr[:, a] @ sr.T) * (dim + rot) ** -0.5).masked_fill(~mask, -math.inf)
            top = torch.maximum(scores.max(-1, keepdim=True).values, w["sink"][a])
            e = torch.exp(scores - top)
            mixed.append((e / (e.sum(-1, keepdim=True) + torch.exp(w["sink"][a] - top))) @ vr[:, a])
        out.append(torch.cat(mixed, dim=1))
    return {"out": torch.cat(out) @ w["o_proj.weight"].T}


# --------------------------------------------------------------------------- the next tokens
def _prepare_sample(case, seed):
    d, rows = _Draw(seed), case["rows"]
    logits = d.normal(rows, case["vocab"], std=2.5, dtype=torch.float32)
    params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"] or None, top_p=case["top_p"], seed=seed + r)
              for r in range(rows)]
    return dict(run=_run_sample, sampler=Sampler(DEVICE, 64), logits=logits, params=params, indices=list(range(rows)))


def _run_sample(s):
    return {"tokens": s["sampler"].sample(s["logits"], s["params"], s["indices"])}


# --------------------------------------------------------------------------- what perf measures with
def prepare(case, seed):
    with torch.inference_mode():
        return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    with torch.inference_mode():
        return state["run"](state)


def exact(case, seed):
    statement = globals().get("_exact_" + case["kind"])     # a draw is a hash of its seed: no 64-bit value
    if statement is None:
        return None
    with torch.inference_mode():
        return statement(case, seed)


def _pairs(lengths, cached=0, window=0):
    """(query, key) pairs that a causal mask leaves."""
    total = 0
    for n in lengths:
        if not window:
            total += n * cached + n * (n + 1) // 2
        else:
            total += sum(min(window, cached + i + 1) for i in range(n))
    return total


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"] + 4 * case["rows"], "flops": 0.0}
    s = SIZES[case["model"]]
    h, ff, heads, kv, size = s["width"], s["ff"], s["heads"], s["kv_heads"], s["size"]
    rows = (heads + 2 * kv) * size
    if kind == "qwen_layer":
        lengths, each = _lengths(case), 4 if case["dtype"] == "float32" else 2
        t, matrices = sum(lengths), h * (rows + heads * size + 3 * ff)
        pairs = _pairs(lengths, case["cached"])
        return {"bytes": each * (matrices + 2 * kv * size * (t + case["cached"] * len(lengths))) + 12.0 * t * h,
                "flops": 2.0 * t * matrices + 4.0 * heads * size * pairs}
    if kind == "qwen_step":
        n, layers = case["requests"], s["layers"]
        matrices = layers * h * (rows + heads * size + 3 * ff) + s["vocab"] * h
        return {"bytes": 2.0 * matrices + 4.0 * n * layers * kv * size * case["context"] + 4.0 * n * s["vocab"],
                "flops": 2.0 * n * matrices + 4.0 * n * layers * heads * size * case["context"]}
    if kind == "lightning":
        lengths = _lengths(case)
        t, matrices, state = sum(lengths), 5 * h * heads * size, heads * size * size
        return {"bytes": 2.0 * matrices + 4.0 * t * h + 8.0 * len(lengths) * state,
                "flops": 2.0 * t * matrices + 4.0 * t * state}
    if kind == "mamba2":
        lengths = _lengths(case)
        inner, n = heads * size, 128
        t, matrices, state = sum(lengths), h * (3 * inner + 2 * n + inner // 64), inner * n
        return {"bytes": 2.0 * matrices + 4.0 * t * h + 8.0 * len(lengths) * (state + 3 * (inner + 2 * n)),
                "flops": 2.0 * t * matrices + 4.0 * t * state}
    if kind == "memory":
        lengths, memory_heads = _lengths(case), heads // 2
        vdim = h // memory_heads
        t = sum(lengths)
        matrices = h * memory_heads * (2 * size + 3 * vdim + 2)
        state = memory_heads * size * (vdim + 1)
        return {"bytes": 2.0 * matrices + 4.0 * t * h + 4.0 * len(lengths) * state, "flops": 2.0 * t * matrices + 4.0 * t * state}
    if kind in ("kanavik_layer", "kanavik_step"):
        matrices = h * (rows + heads * size + 3 * h + 3 * ff + 2 * _SIDE) + 2 * h * h // heads
        if kind == "kanavik_layer":
            lengths = _lengths(case)
            t = sum(lengths)
            pairs = _pairs(lengths, 0, _WINDOW)
            return {"bytes": 2.0 * (matrices + 2 * kv * size * t) + 8.0 * t * h,
                    "flops": 2.0 * t * matrices + (4.0 * heads * size + 2.0 * heads * heads) * pairs}
        n, layers, keys = case["requests"], case["layers"], min(_WINDOW, case["context"])
        everything = layers * matrices + s["vocab"] * h
        return {"bytes": 2.0 * everything + n * layers * (4.0 * kv * size * keys + 80.0 * h) + 4.0 * n * s["vocab"],
                "flops": 2.0 * n * everything + n * layers * keys * (4.0 * heads * size + 2.0 * heads * heads)}
    if kind == "routed":
        t, inner = case["tokens"], ff // case["top"]
        return {"bytes": 2.0 * case["experts"] * 3 * h * inner + 6.0 * t * h,
                "flops": 2.0 * t * (case["top"] * 3 * h * inner + case["experts"] * h)}
    lengths, rank, rot = _lengths(case), case["rank"], case["rot"]
    t = sum(lengths)
    matrices = h * (heads * (size + rot) + rank + rot + heads * size) + 2 * heads * size * rank
    return {"bytes": 2.0 * matrices + 4.0 * t * h + 2.0 * t * (rank + rot),
            "flops": 2.0 * t * matrices + 2.0 * heads * (2 * size + rot) * _pairs(lengths, 0, case["window"])}


def tolerance(case):
    """Four times what each kind showed against its statement in 64 bits, rounded up: rounding of bfloat16 values
    between kernels, and for the 32-bit layer that of its sums."""
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    if kind == "qwen_layer" and case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if kind in ("qwen_step", "kanavik_step"):
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 1.5e-2, "max": 0.3}
