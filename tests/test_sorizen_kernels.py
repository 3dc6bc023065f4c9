"""The kernels that came with the Sorizen decoder, each alone against its plain PyTorch statement, at
sizes other than any model's: the residual streams' write, read and norm in one pass, the store
kernel of latent attention without a query latent, windows, sinks and gates in the attention kernels
over rows that are keys and values at once, the router's groups by their two best scores, the exact
GELU."""
import pytest
import torch

import kernel_references as ref
from test_gpu_kernels import _attention_case, status, tol

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def close(got, want, dtype):
    torch.testing.assert_close(got, want, **(dict(rtol=1e-4, atol=2e-5) if dtype == torch.float32 else tol(dtype)))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("streams", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("tokens, hidden, splits", [
    (1, 64, 1), (5, 320, 7), (9, 100, 20), (6, 37, 3), (200, 48, 1), (333, 1000, 1), (150, 1536, 1), (12, 2500, 16),
    (140, 4096, 1), (3, 5000, 2), (150, 51, 1),
])
def test_streams_write_read_and_norm(dev, dtype, streams, tokens, hidden, splits):
    """Few rows with partial sums, many rows, widths no vector fits; the first write makes the streams of one
    row, later ones work in place; a look at some rows stores nothing."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(1)

    def floats(*shape, scale=1.0, offset=0.0):
        return (offset + scale * torch.randn(shape, generator=gen)).to(dev)

    pending = floats(splits, tokens, hidden) if splits > 1 else floats(tokens, hidden).to(dtype)
    mix, write, read = floats(streams, streams), floats(streams), floats(streams)
    weight, bias = floats(hidden, scale=0.1, offset=1.0), floats(hidden)
    first = floats(tokens, hidden, offset=2.0)
    rows = torch.tensor([tokens - 1, 0, tokens // 2], dtype=torch.int32, device=dev)
    for centre in (True, False):
        results = []
        for fn in (ops.hyper_norm, ref.hyper_norm):
            outs = [torch.full((tokens, hidden), float("nan"), dtype=dtype, device=dev) for _ in range(3)]
            picked = torch.full((3, hidden), float("nan"), dtype=dtype, device=dev)
            made = torch.full((streams, tokens, hidden), float("nan"), device=dev)
            eps = 1e-5
            fn(None, first, streams, None, read, None, weight, bias, centre, eps, outs[0])
            fn(pending, first, streams, (mix, write), read, made, weight, bias if centre else None, centre, eps, outs[1])
            after_first = made.clone()
            fn(pending, made, streams, (mix, write), None, None, weight, bias, centre, eps, picked, rows)
            assert torch.equal(made, after_first)
            fn(pending, made, streams, (mix, write), read, made, weight, bias, centre, eps, outs[2])
            results.append((*outs, picked, after_first, made))
        for got, want in zip(*results):
            close(got, want, got.dtype if got.dtype == torch.bfloat16 else torch.float32)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens, hidden", [(7, 64), (300, 768), (5, 33)])
def test_layer_norm_on_one_plain_stream(dev, dtype, tokens, hidden):
    """The norm part as a model with one stream uses it: the pending output is added to the residual."""
    from einf_b200.config.specs import PartSpec
    from einf_b200.parts.base import Runtime, build_part

    gen = torch.Generator().manual_seed(2)
    w, b = 1 + 0.1 * torch.randn(hidden, generator=gen), torch.randn(hidden, generator=gen)
    norm = build_part("norm", PartSpec("layernorm", {"size": hidden, "eps": 1e-5}), {"weight": w, "bias": b},
                      Runtime(dtype, dev))
    residual = (3 + torch.randn((tokens, hidden), generator=gen)).to(dev)
    pending = torch.randn((tokens, hidden), generator=gen).to(dtype).to(dev)
    total = residual + pending.float()
    want = torch.nn.functional.layer_norm(total, (hidden,), w.to(dev), b.to(dev), 1e-5)
    rows = torch.tensor([tokens - 1, 1], dtype=torch.int32, device=dev)
    before = residual.clone()
    close(norm.forward(pending, residual, rows=rows), want[rows.long()].to(dtype), dtype)
    assert torch.equal(residual, before)
    close(norm.forward(pending, residual), want.to(dtype), dtype)
    close(residual, total, torch.float32)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, dim, rot, rank, row, interleaved, gated", [
    (4, 16, 8, 24, 32, True, True), (3, 12, 4, 20, 24, True, False), (6, 32, 16, 40, 64, False, True),
    (1, 8, 2, 8, 10, True, True), (12, 64, 32, 96, 128, True, False), (16, 128, 64, 512, 576, True, True),
])
@pytest.mark.parametrize("tokens, splits", [(9, 1), (9, 5), (310, 1)])
def test_latent_store_without_a_query_latent(dev, dtype, heads, dim, rot, rank, row, interleaved, gated, tokens, splits):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(3)
    page, pages = 4, 90
    width = rank + rot + heads * (dim + rot) + (heads if gated else 0) + 3       # three elements no one looks at
    if splits == 1:
        product = torch.randn((tokens, width), generator=gen).to(dtype).to(dev)
    else:
        product = torch.randn((splits, tokens, width), generator=gen).to(dev)
    slots = torch.randperm(page * pages, generator=gen)[:tokens].to(torch.int32)
    slots[2] = -1
    slots = slots.to(dev)
    positions = torch.randint(0, 3000, (tokens,), generator=gen).to(torch.int32).to(dev)
    inv_freq = (5000.0 ** (-torch.arange(rot // 2) / (rot // 2))).float().to(dev)
    norm = (1 + 0.1 * torch.randn(rank, generator=gen)).to(dev)
    for copied in (True, False):
        results = []
        st = status(dev)
        for fn in (ops.latent_qkv_store, ref.latent_qkv_store):
            plain = torch.zeros((tokens, heads, dim), dtype=dtype, device=dev) if copied else None
            full = torch.full((tokens, heads, row), 7.0, dtype=dtype, device=dev)
            full[:, :, rank:] = float("nan")                # all of it is written
            gate = torch.zeros((tokens, heads), device=dev) if gated else None
            cache = torch.full((pages, 1, page, row), 5.0, dtype=dtype, device=dev)
            fn(product, rank, rot, norm, 1e-5, positions, inv_freq, interleaved, 1.21, slots, plain, full, gate, cache, st,
               dim)
            results.append([t for t in (plain, full, gate, cache) if t is not None])
        assert int(st) == 0
        for got, want in zip(*results):
            close(got, want, got.dtype if got.dtype == torch.bfloat16 else torch.float32)
        assert bool((results[0][1 if copied else 0][:, :, :rank] == 7.0).all())      # the absorbed part is someone else's
    slots[1] = page * pages + 3                             # beyond the pool: reported, not written
    rows, part = torch.empty((tokens, rank), dtype=dtype, device=dev), torch.empty((tokens, rot), dtype=dtype, device=dev)
    again = torch.zeros_like(cache)
    ops.latent_qkv_store(product, rank, rot, norm, 1e-5, positions, inv_freq, interleaved, 1.0, slots, None, torch.empty_like(full),
                         gate, again, st, dim, rows=rows, part=part)
    want = [torch.empty_like(rows), torch.empty_like(part)]      # the cache rows' two parts, bit for bit
    if dtype == torch.bfloat16 and rank % 8 == 0 and rot % 8 == 0 and again.shape[3] % 8 == 0:
        ops.latent_rows(again, slots, *want)
        assert torch.equal(rows, want[0]) and torch.equal(part, want[1])
    ops.latent_qkv_store(product, rank, rot, norm, 1e-5, positions, inv_freq, interleaved, 1.0, slots, None, full, gate,
                         cache, st, dim)
    assert int(st) == ops.STATUS_BAD_PAGE


def sink_and_gate(dev, heads, tokens):
    gen = torch.Generator().manual_seed(4)
    sink = (torch.randn(heads, generator=gen) * 3).to(dev)
    sink[0], sink[-1] = 40.0, -40.0          # nearly all of the weight; as good as absent
    return sink, torch.rand((tokens, heads), generator=gen).to(dev)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, rank, rot, page_size", [(3, 24, 8, 4), (18, 96, 48, 16), (5, 512, 64, 16), (1, 9, 2, 8)])
@pytest.mark.parametrize("window", [None, 1, 33, 150])
def test_shared_row_decode_with_window_sink_and_gate(dev, dtype, heads, rank, rot, page_size, window):
    from einf_b200 import ops

    row = rank + rot
    requests = [(0, 1), (page_size * 4 - 1, 1), (31, 1), (32, 1), (33, 1), (149, 1), (150, 1), (700, 1)]
    (q, k, _, table, seq, pos), _, _ = _attention_case(dev, dtype, heads, 1, row, page_size, requests, window)
    sink, gate = sink_and_gate(dev, heads, q.shape[0])
    scale = 2.0 * row ** -0.5
    for splits in (1, 3, 8):
        for s, g in ((sink, None), (None, gate), (sink, gate)):
            out = torch.full((q.shape[0], heads, rank), float("nan"), dtype=dtype, device=dev)
            want = torch.empty_like(out)
            st = status(dev)
            ops.latent_decode_attention(q, k, table, seq, pos, out, scale, splits, st, window, s, g)
            ref.latent_decode_attention(q, k, table, seq, pos, want, scale, splits, st, window, s, g)
            assert int(st) == 0
            close(out, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, rank, rot", [(3, 24, 8), (4, 512, 64)])
@pytest.mark.parametrize("window", [None, 5])
def test_general_attention_with_a_gate(dev, dtype, heads, rank, rot, window):
    from einf_b200 import ops

    requests = [(0, 1), (0, 8), (3, 6), (15, 6), (70, 1), (0, 37)]
    (q, k, _, table, seq, pos), scale, _ = _attention_case(dev, dtype, heads, 1, rank + rot, 4, requests, window)
    sink, gate = sink_and_gate(dev, heads, q.shape[0])
    out = torch.full((q.shape[0], heads, rank), float("nan"), dtype=dtype, device=dev)
    want = torch.empty_like(out)
    st = status(dev)
    ops.paged_attention_generic(q, k, None, table, seq, pos, out, scale, window, st, values_in_keys=rank, sink=sink, gate=gate)
    ref.paged_attention_generic(q, k, None, table, seq, pos, want, scale, window, st, values_in_keys=rank, sink=sink, gate=gate)
    assert int(st) == 0
    close(out, want, dtype)


@pytest.mark.parametrize("size", [64, 128])
@pytest.mark.parametrize("heads", [1, 6, 18])
@pytest.mark.parametrize("window", [None, 40, 1000])
def test_tensor_core_attention_with_a_gate(dev, size, heads, window):
    """Row tiles alone and clusters that share one, single tokens in one cluster and in several."""
    from einf_b200 import ops

    dtype = torch.bfloat16
    requests = [(0, 130), (2100, 70), (0, 5), (1500, 1), (63, 1), (0, 1)]
    (q, k, _, table, seq, pos), scale, _ = _attention_case(dev, dtype, heads, 1, size, 16, requests, window)
    sink, gate = sink_and_gate(dev, heads, q.shape[0])
    want = torch.zeros((q.shape[0], heads, size), dtype=dtype, device=dev)
    st = status(dev)
    ref.paged_attention_generic(q, k, k, table, seq, pos, want, scale, window, st, sink=sink, gate=gate)
    tiles, token = [], 0
    singles = []
    for r, (start, n) in enumerate(requests):
        if n == 1:
            singles.append(token)
        else:
            for at in range(0, n, 128):
                tiles.append([r, token + at, min(128, n - at), start + at])
        token += n
    tiles = torch.tensor(tiles, dtype=torch.int32, device=dev)
    single_tokens = torch.tensor(singles, dtype=torch.int32, device=dev)
    for cluster in (1, 4):
        out = torch.zeros_like(want)
        ops.paged_prefill_attention(q, k, k, table, tiles, out, scale, window, st, prefill_cluster=cluster, sink=sink,
                                    gate=gate)
        for clusters, splits in ((1, 1), (4, 1), (2, 2)):
            ops.paged_decode_attention_tcgen05(q, k, k, table, seq, pos, out, scale, window, clusters, st, single_tokens,
                                               splits, sink=sink, gate=gate)
            torch.testing.assert_close(out, want, rtol=3e-2, atol=2e-2)
    assert int(st) == 0


@pytest.mark.parametrize("experts, top, groups", [
    (15, 2, (3, 2)), (12, 4, (4, 2)), (9, 3, (3, 1)), (8, 8, (4, 4)), (6, 2, (6, 3)), (5, 2, None), (1, 1, (1, 1)),
    (160, 8, (40, 5)), (64, 6, (2, 1)),
])
@pytest.mark.parametrize("score", ["sigmoid", "softmax"])
@pytest.mark.parametrize("corrected", [False, True])
def test_router_with_groups_by_their_two_best(dev, experts, top, groups, score, corrected):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(5)
    logits = (torch.randn((43, experts), generator=gen) * 2).to(dev)
    correction = (torch.randn(experts, generator=gen) * 0.2).to(dev) if corrected else None
    results = []
    for fn in (ops.router_topk, ref.router_topk):
        ids = torch.zeros((43, top), dtype=torch.int32, device=dev)
        weights = torch.zeros((43, top), dtype=torch.float32, device=dev)
        fn(logits, top, score, True, ids, weights, experts, correction, groups, group_best=2, renormalise_eps=0.25,
           weight_scale=1.75)
        results.append((ids, weights))
    assert torch.equal(results[0][0], results[1][0])
    torch.testing.assert_close(results[0][1], results[1][1], rtol=1e-5, atol=1e-7)
    # written out for a few rows
    scores = (torch.softmax(logits, dim=-1) if score == "softmax" else torch.sigmoid(logits)).double().cpu()
    choice = scores + (0 if correction is None else correction.double().cpu())
    for t in range(6):
        chosen = results[0][0][t].tolist()
        if groups is not None:
            per = experts // groups[0]
            pairs = [sum(sorted(choice[t, g * per:(g + 1) * per].tolist())[-2:]) for g in range(groups[0])]
            kept = set(sorted(range(groups[0]), key=lambda g: -pairs[g])[:groups[1]])
            assert {e // per for e in chosen} <= kept
        total = sum(float(scores[t, e]) for e in chosen) + 0.25
        for j, e in enumerate(chosen):
            assert float(results[0][1][t, j]) == pytest.approx(1.75 * float(scores[t, e]) / total, rel=1e-5)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("splits", [1, 3])
def test_exact_gelu(dev, dtype, splits):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(6)
    x = (3 * torch.randn((splits, 11, 56), generator=gen)).to(dev)
    x = x if splits > 1 else x[0].to(dtype)
    out = torch.empty((11, 56), dtype=dtype, device=dev)
    ops.activation(x, out, "gelu")
    z = x.double().sum(0) if splits > 1 else x.double()
    want = torch.nn.functional.gelu(z)
    close(out, want.to(dtype), dtype)


@pytest.mark.parametrize("heads, rank, rot, row", [
    (1, 50, 14, 64), (7, 136, 24, 192), (18, 300, 20, 320), (12, 512, 64, 576), (130, 96, 32, 128), (5, 400, 48, 448),
    (3, 600, 40, 640),
])
@pytest.mark.parametrize("page_size", [8, 16, 64])
@pytest.mark.parametrize("window", [None, 1, 40, 1000])
def test_latent_attention_on_the_tensor_cores(dev, heads, rank, rot, row, page_size, window):
    """Portions beside single tokens, rows longer than what they hold, values in one and in two parts, keys in shares."""
    from einf_b200 import ops

    dtype = torch.bfloat16
    requests = [(0, 131), (1100, 70), (0, 5), (1500, 1), (63, 1), (0, 1), (200, 2)]
    (q, k, _, table, seq, pos), _, _ = _attention_case(dev, dtype, heads, 1, row, page_size, requests, window)
    q[:, :, rank + rot:] = 0
    k[..., rank + rot:] = 0
    sink, gate = sink_and_gate(dev, heads, q.shape[0])
    scale = 2.0 * (rank + rot) ** -0.5
    tiles, singles, token = [], [], 0
    for r, (start, n) in enumerate(requests):
        if n == 1:
            singles.append(token)
        for at in range(0, n if n > 1 else 0, 128):
            tiles.append([r, token + at, min(128, n - at), start + at])
        token += n
    tiles = torch.tensor(tiles, dtype=torch.int32, device=dev)
    listed = torch.tensor(singles, dtype=torch.int32, device=dev)
    for s, g in ((None, None), (sink, gate)):
        st = status(dev)
        want = torch.zeros((q.shape[0], heads, rank), dtype=dtype, device=dev)
        ref.paged_attention_generic(q, k, None, table, seq, pos, want, scale, window, st, values_in_keys=rank, sink=s, gate=g)
        for longest in (100, 1501):           # the longest context sets the number of shares
            out = torch.full((q.shape[0], heads, rank), float("nan"), dtype=dtype, device=dev)
            ops.latent_attention(q, k, table, seq, pos, tiles, listed, len(singles), out, scale, window, st,
                                 max_context=longest, sink=s, gate=g)
            torch.testing.assert_close(out, want, rtol=3e-2, atol=2e-2)
        # the same single tokens alone, as a decode step has them
        picked = [t[listed.long()].contiguous() for t in (q, seq, pos)]
        alone = torch.full((len(singles), heads, rank), float("nan"), dtype=dtype, device=dev)
        ops.latent_attention(picked[0], k, table, picked[1], picked[2], None, None, len(singles), alone, scale, window, st,
                             max_context=1501, sink=s, gate=None if g is None else g[listed.long()].contiguous())
        assert torch.equal(alone, out[listed.long()])
        assert int(st) == 0


def test_latent_attention_reports_a_page_outside_the_pool(dev):
    from einf_b200 import ops

    (q, k, _, table, seq, pos), scale, _ = _attention_case(dev, torch.bfloat16, 4, 1, 192, 16, [(0, 60)], None)
    table[0, 2] = k.shape[0] + 5              # reported, not read
    st = status(dev)
    out = torch.zeros((60, 4, 128), dtype=torch.bfloat16, device=dev)
    tiles = torch.tensor([[0, 0, 60, 0]], dtype=torch.int32, device=dev)
    ops.latent_attention(q, k, table, seq, pos, tiles, None, 0, out, scale, None, st)
    assert int(st) == ops.STATUS_BAD_PAGE and torch.isfinite(out).all()


@pytest.mark.parametrize("heads, dim, rot, value", [(3, 128, 64, 128), (2, 64, 64, 64), (1, 40, 24, 72), (5, 136, 8, 8), (2, 16, 0, 128)])
@pytest.mark.parametrize("window", [None, 5, 100])
@pytest.mark.parametrize("lengths", [(2,), (63, 64, 65), (130, 2, 257)])
@pytest.mark.parametrize("options", [False, True])
def test_prompts_head_by_head(dev, heads, dim, rot, value, window, lengths, options):
    """Prompts with keys and values of their own per head against the plain statement in 64 bits: lengths around the
    kernel's tiles of 64 and the tiles of 128 it is given, keys that fill no tile of 64 elements, views of wider rows."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim + sum(lengths))
    tokens = sum(lengths)
    draw = lambda *shape: torch.randn(shape, generator=gen).to(torch.bfloat16).to(dev)  # noqa: E731
    wide, kv = draw(tokens, heads, dim + rot + 8), draw(tokens, heads * (dim + value) + 8)
    q_plain, q_rot = wide[:, :, :dim], draw(tokens, heads, rot + 16)[:, :, 8:8 + rot]
    k_plain = kv[:, :heads * dim].unflatten(1, (heads, dim))
    v = kv[:, heads * dim:heads * (dim + value)].unflatten(1, (heads, value))
    k_rot = draw(tokens, rot)
    sink = torch.randn(heads, generator=gen).to(dev) if options else None
    gate = torch.rand((tokens, heads), generator=gen).to(dev) if options else None
    tiles, first = [], 0
    for r, n in enumerate(lengths):
        tiles += [(r, first + at, min(128, n - at), at) for at in range(0, n, 128)]
        first += n
    out = torch.full((tokens, heads, value), float("nan"), dtype=torch.bfloat16, device=dev)
    scale = (dim + rot) ** -0.5
    ops.head_prompt_attention(q_plain, q_rot, k_plain, k_rot, v, torch.tensor(tiles, dtype=torch.int32, device=dev), out, scale,
                              window, sink=sink, gate=gate)
    first = 0
    for n in lengths:
        part = slice(first, first + n)
        scores = torch.einsum("ihd,jhd->hij", q_plain[part].double(), k_plain[part].double())
        scores = (scores + torch.einsum("ihr,jr->hij", q_rot[part].double(), k_rot[part].double())) * scale
        i, j = torch.arange(n, device=dev)[:, None], torch.arange(n, device=dev)[None, :]
        seen = (j <= i) if window is None else (j <= i) & (j > i - window)
        scores = scores.masked_fill(~seen, float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink[:, None, None].expand(heads, n, 1)], dim=2)
        weights = torch.softmax(scores, dim=2)[:, :, :n]
        want = torch.einsum("hij,jhv->ihv", weights, v[part].double())
        size = torch.einsum("hij,jhv->ihv", weights, v[part].double().abs())
        if gate is not None:
            want, size = want * gate[part][:, :, None], size * gate[part][:, :, None]
        # the output's rounding, the weights' (each to bfloat16), and 2^-16 of the terms' sizes for scores, exponentials and sums
        bound = 2.0 ** -8 * want.abs() + (2.0 ** -8 + 2.0 ** -16) * size
        assert bool(((out[part].double() - want).abs() <= bound).all())
        first += n


@pytest.mark.parametrize("heads, dim, value, window, lengths", [
    (3, 128, 128, None, (700, 129, 1)), (2, 64, 64, 200, (900,)), (1, 128, 64, None, (256, 384)), (2, 64, 128, 130, (385, 5))])
def test_prompts_head_by_head_in_tensor_memory(dev, heads, dim, value, window, lengths):
    """Prompts of many key tiles, both groups' turns and one group's alone, scores that grow along the prompt (so that the
    rows' references move), and values that are not finite in the request behind, whose rows fill up the last tile."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim + value)
    tokens, rot = sum(lengths), 64
    draw = lambda *shape: torch.randn(shape, generator=gen).to(torch.bfloat16).to(dev)  # noqa: E731
    q_plain, q_rot, k_rot, v = draw(tokens, heads, dim), draw(tokens, heads, rot), draw(tokens, rot), draw(tokens, heads, value)
    grow = torch.cat([torch.linspace(0.1, 8.0, n) for n in lengths])[:, None, None].to(dev)
    k_plain = (draw(tokens, heads, dim).float() * grow).to(torch.bfloat16)
    tiles, first = [], 0
    for r, n in enumerate(lengths):
        tiles += [(r, first + at, min(128, n - at), at) for at in range(0, n, 128)]
        first += n
    tiles, scale = torch.tensor(tiles, dtype=torch.int32, device=dev), (dim + rot) ** -0.5
    out, status = torch.full((tokens, heads, value), float("nan"), dtype=torch.bfloat16, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    ops.head_prompt_attention(q_plain, q_rot, k_plain, k_rot, v, tiles, out, scale, window, status=status, tensor_memory=True)
    first = 0
    for n in lengths:
        part = slice(first, first + n)
        scores = torch.einsum("ihd,jhd->hij", q_plain[part].double(), k_plain[part].double())
        scores = (scores + torch.einsum("ihr,jr->hij", q_rot[part].double(), k_rot[part].double())) * scale
        i, j = torch.arange(n, device=dev)[:, None], torch.arange(n, device=dev)[None, :]
        scores = scores.masked_fill(~((j <= i) & (j > i - (window or tokens))), float("-inf"))
        weights = torch.softmax(scores, dim=2)
        want = torch.einsum("hij,jhv->ihv", weights, v[part].double())
        size = torch.einsum("hij,jhv->ihv", weights, v[part].double().abs())
        bound = 2.0 ** -8 * want.abs() + (2.0 ** -8 + 2.0 ** -14) * size      # as above; scores of up to fifty
        assert bool(((out[part].double() - want).abs() <= bound).all())
        first += n
    if len(lengths) > 1:
        again, begin = torch.empty_like(out), lengths[0]
        v[begin:], k_plain[begin:] = float("inf"), float("nan")
        ops.head_prompt_attention(q_plain, q_rot, k_plain, k_rot, v, tiles, again, scale, window, status=status, tensor_memory=True)
        assert torch.equal(again[:begin], out[:begin])
    assert int(status) == 0


def _prompt_in_64_bits(q_plain, q_rot, k_plain, k_rot, v, scale, window):
    """Which keys a row sees, and the rows' results with values that are not finite left out."""
    n = q_plain.shape[0]
    scores = torch.einsum("ihd,jhd->hij", q_plain.double(), k_plain.double())
    scores = (scores + torch.einsum("ihr,jr->hij", q_rot.double(), k_rot.double())) * scale
    i, j = torch.arange(n, device=v.device)[:, None], torch.arange(n, device=v.device)[None, :]
    seen = (j <= i) & (j > i - (window or n))
    weights = torch.softmax(scores.masked_fill(~seen, float("-inf")), dim=2)
    return seen, torch.einsum("hij,jhv->ihv", weights, torch.nan_to_num(v.double(), 0.0, 0.0, 0.0))


def _prompt_tiles(n, dev):
    return torch.tensor([(0, at, min(128, n - at), at) for at in range(0, n, 128)], dtype=torch.int32, device=dev)


@pytest.mark.parametrize("tensor_memory", [True, False])
@pytest.mark.parametrize("dim, value, window", [(64, 64, None), (128, 128, 100)])
def test_scores_that_are_not_finite_are_not_hidden(dev, tensor_memory, dim, value, window):
    """A row that sees a score which is NaN or plus infinity is NaN, and no other row is: NaN in a key, an infinite key
    (plus or minus infinite scores, by the query's sign), NaN in a query; in the first, the last and a middle tile."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim)
    heads, rot, n, scale = 2, 64, 300, (dim + 64) ** -0.5
    draw = lambda *shape: torch.randn(shape, generator=gen).to(torch.bfloat16).to(dev)  # noqa: E731
    q_plain, q_rot, k_plain, k_rot, v = draw(n, heads, dim), draw(n, heads, rot), draw(n, heads, dim), draw(n, rot), draw(n, heads, value)
    tiles, status = _prompt_tiles(n, dev), torch.zeros(1, dtype=torch.int32, device=dev)
    for where in (5, 130, 290):
        q, k = q_plain.clone(), k_plain.clone()
        k[where, 0, 3] = float("nan")
        k[where - 3, 1, 7] = float("inf")
        q[where - 2, 1, 0] = float("nan")
        out = torch.zeros((n, heads, value), dtype=torch.bfloat16, device=dev)
        ops.head_prompt_attention(q, q_rot, k, k_rot, v, tiles, out, scale, window, status=status, tensor_memory=tensor_memory)
        want = _prompt_in_64_bits(q, q_rot, k, k_rot, v, scale, window)[1]
        assert torch.equal(out.isnan(), want.isnan()) and 0 < int(want.isnan().sum()) < want.numel()
        fine = ~want.isnan()
        torch.testing.assert_close(out[fine].double(), want[fine], rtol=2e-2, atol=2e-2)
    assert int(status) == 0


@pytest.mark.parametrize("scale, heads_first", [(0.0, False), (-0.1, False), (0.1, True)])
def test_prompts_that_the_tensor_memory_kernel_leaves_to_the_other(dev, scale, heads_first):
    """Scores that a factor turns round or levels, and heads farther apart than tokens."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(3)
    heads, dim, rot, value, n = 2, 64, 64, 64, 200

    def draw(*shape):
        t = torch.randn(shape, generator=gen).to(torch.bfloat16).to(dev)
        return t.transpose(0, 1).contiguous().transpose(0, 1) if heads_first and len(shape) == 3 else t

    q_plain, q_rot, k_plain, k_rot, v = draw(n, heads, dim), draw(n, heads, rot), draw(n, heads, dim), draw(n, rot), draw(n, heads, value)
    out, status = torch.zeros((n, heads, value), dtype=torch.bfloat16, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    ops.head_prompt_attention(q_plain, q_rot, k_plain, k_rot, v, _prompt_tiles(n, dev), out, scale, None, status=status)
    want = _prompt_in_64_bits(q_plain, q_rot, k_plain, k_rot, v, scale, None)[1]
    torch.testing.assert_close(out.double(), want, rtol=2e-2, atol=2e-2)
    assert int(status) == 0


@pytest.mark.parametrize("value, window", [(64, None), (128, 100), (64, 130)])
def test_values_that_are_not_finite_stay_with_the_rows_that_see_them(dev, value, window):
    """Infinite and NaN values in a prompt on the tensor cores: the columns of the rows that see them, and nothing else."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(value)
    heads, dim, rot, n, scale = 2, 64, 64, 301, 0.1
    draw = lambda *shape: torch.randn(shape, generator=gen).to(torch.bfloat16).to(dev)  # noqa: E731
    q_plain, q_rot, k_plain, k_rot, v = draw(n, heads, dim), draw(n, heads, rot), draw(n, heads, dim), draw(n, rot), draw(n, heads, value)
    v[100, 0, 3], v[127, 0, value - 1], v[128, 1, 0], v[200, 1, 0] = float("inf"), -float("inf"), float("nan"), float("inf")
    v[300, 1, 33], v[150, 0, 3] = float("inf"), -float("inf")
    out, status = torch.zeros((n, heads, value), dtype=torch.bfloat16, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    ops.head_prompt_attention(q_plain, q_rot, k_plain, k_rot, v, _prompt_tiles(n, dev), out, scale, window, status=status,
                              tensor_memory=True)
    seen, want = _prompt_in_64_bits(q_plain, q_rot, k_plain, k_rot, v, scale, window)
    for token, head, column in (~torch.isfinite(v)).nonzero().tolist():
        want[seen[:, token], head, column] += v[token, head, column].double()
    torch.testing.assert_close(out.double(), want, rtol=2e-2, atol=2e-2, equal_nan=True)
    assert int(status) == 0


@pytest.mark.parametrize("heads, dim, rot, value, rank, q_rank, page", [
    (3, 128, 64, 128, 512, None, 16), (4, 40, 24, 72, 32, 64, 16), (2, 64, 16, 64, 192, 40, 8), (2, 64, 8, 40, 176, 40, 5)])
@pytest.mark.parametrize("window", [None, 60])
def test_a_prompt_gets_what_it_gets_beside_prompts(dev, heads, dim, rot, value, rank, q_rank, page, window):
    """A latent layer's prompts that start in a step are bit for bit the same beside single tokens and portions that go on as
    beside a prompt of as many tokens that starts with them (equal counts: equal products); and those others are
    what a layer that runs everything on the rows makes of them."""
    from einf_b200 import ops
    from einf_b200.config.specs import PartSpec
    from einf_b200.engine.batch import StepInputBuilder
    from einf_b200.parts.base import CacheView, Runtime, build_part, part_class, walk_part_specs
    from types import SimpleNamespace

    gen = torch.Generator().manual_seed(rank + rot)
    hidden = 128
    spec = PartSpec("latent_attention", {
        "hidden_size": hidden, "num_heads": heads, "head_size": dim, "rotary_size": rot, "value_head_size": value,
        "kv_rank": rank, "q_rank": q_rank, "scale": (dim + rot) ** -0.5, "eps": 1e-6, "window": window, "sink": True,
        "position": PartSpec("rope", {"rotary_dim": rot, "theta": 1e4})})
    draw = lambda *shape: (torch.randn(shape, generator=gen) * shape[-1] ** -0.5).to(torch.bfloat16).to(dev)  # noqa: E731
    tensors = {"kv_down.weight": draw(rank + rot, hidden), "k_up.weight": draw(heads * dim, rank), "v_up.weight": draw(heads * value, rank),
               "o_proj.weight": draw(hidden, heads * value), "sink": torch.randn(heads, generator=gen).to(dev),
               "kv_norm.weight": torch.ones(rank, dtype=torch.bfloat16, device=dev)}
    if q_rank:
        tensors.update({"q_down.weight": draw(q_rank, hidden), "q_up.weight": draw(heads * (dim + rot), q_rank),
                        "q_norm.weight": torch.ones(q_rank, dtype=torch.bfloat16, device=dev)})
    else:
        tensors["q_proj.weight"] = draw(heads * (dim + rot), hidden)
    runtime = Runtime(torch.bfloat16, dev)
    names = []
    for category, nested in walk_part_specs("mixer", spec):
        names += part_class(category, nested.kind).kernel_libraries(nested, runtime)
    ops.ensure_built(tuple(dict.fromkeys(names)))
    part = build_part("mixer", spec, tensors, runtime)
    assert part.by_heads
    fresh, others = [(0, 150), (0, 2), (0, 64)], [(40, 1), (70, 33), (300, 1), (129, 140), (0, 1)]
    count, rest = sum(n for _, n in fresh), sum(n for _, n in others)
    x = torch.randn((count + rest, hidden), generator=gen).to(torch.bfloat16).to(dev)

    def run(requests):
        needs = [-(-(start + n) // page) for start, n in requests]
        order = torch.randperm(sum(needs), generator=torch.Generator().manual_seed(1)).tolist()
        cache = torch.randn((sum(needs), 1, page, part.row), generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).to(dev)
        builder = StepInputBuilder(dev, page, [sum(needs)], [window], 1000, max(needs), x.shape[0], len(requests))
        ctx, _ = builder.build([SimpleNamespace(input_token_ids=[1] * n, start_position=start, need_sample=False,
                                                block_tables=[[order.pop() for _ in range(need)]])
                                for (start, n), need in zip(requests, needs)])
        out = part.forward(x, ctx, CacheView(group=0, k=cache, v=None, writes=True, page_size=page))
        assert int(ctx.status) == 0
        return out.float().sum(dim=0) if out.dim() == 3 else out.float()

    mixed, together = run(fresh + others), run(fresh + [(0, rest)])
    part.by_heads = False
    on_rows = run(fresh + others)
    assert torch.equal(mixed[:count], together[:count]) and torch.equal(mixed[count:], on_rows[count:])
    assert not torch.equal(mixed[:count], on_rows[:count])                  # the two ways round in different places
    torch.testing.assert_close(mixed[:count], on_rows[:count], rtol=2e-2, atol=2e-2)


def test_latent_rows(dev):
    """Cached rows taken apart, a token without a slot among them."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(3)
    cache = torch.randn((5, 1, 8, 96), generator=gen).to(torch.bfloat16).to(dev)
    slots = torch.tensor([39, 0, -1, 17, 8], dtype=torch.int32, device=dev)
    rows, rest = (torch.full((5, n), float("nan"), dtype=torch.bfloat16, device=dev) for n in (64, 24))
    ops.latent_rows(cache, slots, rows, rest)
    want = cache.view(40, 96)[slots.long().clamp(min=0)]
    want[2] = 0
    assert torch.equal(torch.cat([rows, rest], dim=1), want[:, :88])

