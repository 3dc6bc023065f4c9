"""The score-mixing attention kernels and the gated scan alone, each against its plain PyTorch
statement, at sizes other than any model's: both attention kernels (a CTA per token; the tiled one
with and without its keys split), steps of prompt portions beside single tokens, windows whose edge
falls inside a tile, and the scan in one piece and in segments."""
import pytest
import torch

import kernel_references as ref
from test_gpu_kernels import _attention_case, status, tol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def _step_split(requests):
    """q_tiles and the indices of single tokens for requests given as (start, q_len)."""
    tiles, singles, token = [], [], 0
    for r, (start, q_len) in enumerate(requests):
        if q_len == 1:
            singles.append(token)
        else:
            for first in range(0, q_len, 128):
                tiles.append((r, token + first, min(128, q_len - first), start + first))
        token += q_len
    return (torch.tensor(tiles, dtype=torch.int32).view(-1, 4), torch.tensor(singles, dtype=torch.int32))


def _mixing(heads, generator, dev):
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)])
    talk = torch.eye(heads) + 0.3 * torch.randn((heads, heads), generator=generator)
    sink = torch.randn((heads,), generator=generator)
    return slopes.to(dev), talk.to(dev), sink.to(dev)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, kv_heads, size, vsize, page_size", [
    (4, 2, 16, 16, 4), (3, 1, 32, 24, 8), (14, 2, 64, 64, 16), (6, 3, 48, 40, 16), (8, 8, 128, 128, 16),
    (5, 5, 20, 100, 3), (1, 1, 64, 8, 64), (17, 1, 8, 36, 16), (32, 4, 64, 64, 16),
])
@pytest.mark.parametrize("window", [None, 5, 70])
@pytest.mark.parametrize("parts", ["all", "no sink", "plain"])
def test_tiled_score_mixing_attention(dev, dtype, heads, kv_heads, size, vsize, page_size, window, parts):
    from einf_b200 import ops

    if parts != "all" and (window != 70 or dtype != torch.float32):
        pytest.skip("the optional parts are switched off in one setting")
    requests = [(0, 1), (0, 2 * page_size), (3, 6), (15, 2), (page_size * 4 - 1, 1), (200, 1), (0, 137), (61, 19),
                (130, 70)]
    (q, k, v, table, seq, pos), scale, window = _attention_case(dev, dtype, heads, kv_heads, size, page_size, requests, window)
    generator = torch.Generator().manual_seed(5)
    v = torch.randn((*v.shape[:3], vsize), generator=generator).to(dtype).to(dev)
    slopes, talk, sink = _mixing(heads, generator, dev)
    if parts == "no sink":
        sink = None
    if parts == "plain":
        slopes = talk = sink = None
    q_tiles, singles = _step_split(requests)
    want = torch.empty((q.shape[0], heads, vsize), dtype=dtype, device=dev)
    st = status(dev)
    ref.paged_attention_mixed(q.cpu(), k.cpu(), v.cpu(), table.cpu(), seq.cpu(), pos.cpu(), want_cpu := want.cpu(), scale,
                              window, *(None if t is None else t.cpu() for t in (slopes, talk, sink)), 0.7, st.cpu())
    close = dict(rtol=2e-4, atol=2e-5) if dtype == torch.float32 else tol(dtype)
    for tiled in (False, True):
        out = torch.full_like(want, float("nan"))
        extra = dict(q_tiles=q_tiles.to(dev), single_tokens=singles.to(dev), num_singles=singles.shape[0],
                     max_context=max(s + n for s, n in requests)) if tiled else {}
        if tiled:
            assert ops.mixed_tiled_rows(heads, kv_heads, size, vsize, False) and ops.mixed_tiled_rows(heads, kv_heads, size, vsize, True)
        ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, window, slopes, talk, sink, 0.7, st, **extra)
        assert int(st) == 0
        torch.testing.assert_close(out.cpu(), want_cpu, **close)


@pytest.mark.parametrize("heads, kv_heads, size, vsize, window", [
    (14, 2, 64, 64, 100), (6, 3, 32, 128, None), (5, 1, 16, 8, 64), (8, 8, 16, 72, 1), (32, 1, 112, 64, 63),
])
@pytest.mark.parametrize("parts", ["all", "no slopes", "no mixing"])
def test_mixing_in_the_queries(dev, heads, kv_heads, size, vsize, window, parts):
    """The kernel with the mixing in the queries and the kernel that mixes scores, on the same portions (rows around the tiles
    of 64, portions behind cached tokens): each off the statement in 64 bits by little more than the output's rounding."""
    from einf_b200 import ops

    requests = [(0, 2), (0, 63), (0, 64), (5, 65), (300, 129), (61, 19)]
    (q, k, v, table, seq, pos), scale, window = _attention_case(dev, torch.bfloat16, heads, kv_heads, size, 16, requests, window)
    generator = torch.Generator().manual_seed(11)
    v = torch.randn((*v.shape[:3], vsize), generator=generator).to(torch.bfloat16).to(dev)
    slopes, talk, sink = _mixing(heads, generator, dev)
    slopes, talk = None if parts == "no slopes" else slopes, None if parts == "no mixing" else talk
    q_tiles, singles = _step_split(requests)
    contexts = [start + n for start, n in requests]
    assert ops.mixed_prompt_takes(q, k, v, q, q_tiles.shape[0], 1, 1)
    outs = []
    for tiles_pay in (True, False):
        out = torch.full((q.shape[0], heads, vsize), float("nan"), dtype=torch.bfloat16, device=dev)
        st = status(dev)
        before = ops.MIXED_PROMPT_CTAS, ops.MIXED_PROMPT_FEW_KEYS
        try:
            ops.MIXED_PROMPT_CTAS, ops.MIXED_PROMPT_FEW_KEYS = (0, 0) if tiles_pay else (1 << 30, 0)
            ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, window, slopes, talk, sink, 0.7, st,
                                      q_tiles=q_tiles.to(dev), single_tokens=singles.to(dev), num_singles=0,
                                      max_context=max(contexts))
        finally:
            ops.MIXED_PROMPT_CTAS, ops.MIXED_PROMPT_FEW_KEYS = before
        assert int(st) == 0
        outs.append(out)
    # 64 bits, request by request
    group = torch.arange(heads, device=dev) // (heads // kv_heads)
    first = 0
    for r, (start, n) in enumerate(requests):
        end, rows = start + n, slice(first, first + n)
        pages = table[r, :-(-end // 16)].long()
        if window is not None:
            pages = pages.clamp(min=0)
        keys = k[pages].transpose(1, 2).reshape(-1, kv_heads, size)[:end].double()[:, group]
        values = v[pages].transpose(1, 2).reshape(-1, kv_heads, vsize)[:end].double()[:, group]
        i = torch.arange(start, end, device=dev)[:, None]
        j = torch.arange(end, device=dev)[None, :]
        raw = torch.einsum("ihd,jhd->hij", q[rows].double(), keys) * scale
        if slopes is not None:
            raw = raw - slopes.double()[:, None, None] * (i - j)
        if talk is not None:
            raw = torch.einsum("hg,gij->hij", talk.double(), raw)
        seen = (j <= i) if window is None else (j <= i) & (i - j < window)
        raw = torch.cat([raw.masked_fill(~seen, float("-inf")), sink.double()[:, None, None].expand(heads, n, 1)], dim=2)
        want = 0.7 * torch.einsum("hij,jhv->ihv", torch.softmax(raw, dim=2)[:, :, :-1], values)
        # bfloat16 rounding of the output: 2^-9 of an element; weights of two bfloat16 parts and 32-bit sums: far below
        for out in outs:
            assert bool(((out[rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all())
        first += n


@pytest.mark.parametrize("heads, kv_heads, size, vsize, n", [
    (14, 2, 64, 64, 1), (16, 1, 128, 128, 1), (4, 4, 16, 24, 1), (20, 2, 64, 64, 5), (32, 4, 32, 128, 4), (24, 8, 16, 8, 2)])
def test_mixed_weights_hold_32_bits(dev, heads, kv_heads, size, vsize, n):
    """Single tokens of up to 16 heads and portions of more, over five keys whose values (chosen one after the other, for the last
    token and the first head of every key head) nearly cancel under the weights, so that what is left shows the weights'
    own rounding.  The bound: the output's rounding (2^-8 of it) and 12 roundings to 32 bits of the sum of the terms' sizes
    (scores below one: a score's sums, exp2 and the sum of values; weights of 16 bits are off by up to 2^-16, 256 of those)."""
    from einf_b200 import ops

    requests = [(5 - n, n)] * 12
    (q, k, v, table, seq, pos), scale, _ = _attention_case(dev, torch.bfloat16, heads, kv_heads, size, 16, requests, None)
    scale, per = scale / 4, heads // kv_heads
    generator = torch.Generator().manual_seed(13)
    v = torch.zeros((*k.shape[:3], vsize), dtype=torch.bfloat16, device=dev)
    group, exact = torch.arange(heads, device=dev) // per, []
    for r in range(len(requests)):
        page = int(table[r, 0])
        keys = k[page].transpose(0, 1)[:5].double()[:, group]
        scores = torch.einsum("ihd,jhd->hij", q[n * r:n * (r + 1)].double(), keys) * scale
        seen = torch.arange(5, device=dev)[None, :] <= torch.arange(5 - n, 5, device=dev)[:, None]
        weights = torch.softmax(scores.masked_fill(~seen, float("-inf")), dim=2)
        last = weights[::per, -1]                                          # [kv_heads, 5]
        v[page, :, 0] = (1 + torch.rand((kv_heads, vsize), generator=generator)).to(torch.bfloat16).to(dev)
        for j in range(1, 4):
            so_far = torch.einsum("gj,gjd->gd", last[:, :j], v[page, :, :j].double())
            v[page, :, j] = (-so_far / last[:, j, None]).to(torch.bfloat16)
        exact.append((weights, v[page].transpose(0, 1)[:5].double()[:, group]))
    q_tiles, singles = _step_split(requests)
    out = torch.full((q.shape[0], heads, vsize), float("nan"), dtype=torch.bfloat16, device=dev)
    st = status(dev)
    assert ops.mixed_single_takes(q, k, v) if n == 1 else ops.mixed_prompt_takes(q, k, v, out, q_tiles.shape[0], None, 5)
    ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, None, None, None, None, 1.0, st, q_tiles=q_tiles.to(dev),
                              single_tokens=singles.to(dev), num_singles=singles.shape[0], max_context=5)
    assert int(st) == 0
    for r, (weights, values) in enumerate(exact):
        want, size_of = (torch.einsum("hij,jhv->ihv", weights, t) for t in (values, values.abs()))
        assert float(want[-1, ::per].abs().max()) < 2.0 ** -14
        error = (out[n * r:n * (r + 1)].double() - want).abs()
        assert bool((error <= 2.0 ** -8 * want.abs() + 12 * 2.0 ** -24 * size_of).all()), float((error / size_of).max() * 2 ** 24)


@pytest.mark.parametrize("heads, kv_heads, size, vsize, window", [
    (14, 2, 64, 64, 100), (16, 1, 128, 128, None), (5, 1, 8, 24, 33), (4, 4, 32, 16, 1), (6, 3, 40, 40, None),
])
@pytest.mark.parametrize("parts, splits", [("all", 1), ("all", 3), ("no slopes", 40), ("no mixing", 1)])
def test_single_tokens_with_their_heads_as_rows(dev, heads, kv_heads, size, vsize, window, parts, splits, monkeypatch):
    """Contexts around the chunks of 32 keys, CTAs without a key among those that share a token's, a list of tokens in an
    order of its own."""
    from einf_b200 import ops

    requests = [(0, 1), (30, 1), (31, 1), (32, 1), (600, 1), (129, 1)]
    (q, k, v, table, seq, pos), scale, window = _attention_case(dev, torch.bfloat16, heads, kv_heads, size, 16, requests, window)
    generator = torch.Generator().manual_seed(12)
    v = torch.randn((*v.shape[:3], vsize), generator=generator).to(torch.bfloat16).to(dev)
    slopes, talk, sink = _mixing(heads, generator, dev)
    slopes, talk = None if parts == "no slopes" else slopes, None if parts == "no mixing" else talk
    assert ops.mixed_single_takes(q, k, v)
    monkeypatch.setattr(ops, "mixed_tiled_splits", lambda *_: splits)
    singles = torch.tensor([4, 0, 3, 1, 5], dtype=torch.int32, device=dev)
    out = torch.full((q.shape[0], heads, vsize), float("nan"), dtype=torch.bfloat16, device=dev)
    st = status(dev)
    ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, window, slopes, talk, sink, 0.7, st,
                              q_tiles=torch.empty((0, 4), dtype=torch.int32, device=dev), single_tokens=singles,
                              num_singles=5, max_context=601)
    assert int(st) == 0 and bool(out[2].isnan().all())
    group = torch.arange(heads, device=dev) // (heads // kv_heads)
    for t in singles.tolist():
        end = requests[t][0] + 1
        pages = table[t, :-(-end // 16)].long().clamp(min=0)
        keys = k[pages].transpose(1, 2).reshape(-1, kv_heads, size)[:end].double()[:, group]
        values = v[pages].transpose(1, 2).reshape(-1, kv_heads, vsize)[:end].double()[:, group]
        away = end - 1 - torch.arange(end, device=dev)
        raw = torch.einsum("hd,jhd->hj", q[t].double(), keys) * scale
        if slopes is not None:
            raw = raw - slopes.double()[:, None] * away
        if talk is not None:
            raw = talk.double() @ raw
        if window is not None:
            raw = raw.masked_fill(away >= window, float("-inf"))
        weights = torch.softmax(torch.cat([raw, sink.double()[:, None]], dim=1), dim=1)[:, :-1]
        want = 0.7 * torch.einsum("hj,jhv->hv", weights, values)
        # the output's rounding, 2^-9 of an element; weights of two bfloat16 parts and 32-bit sums: far below
        assert bool(((out[t].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all())


@pytest.mark.parametrize("batch, context, window", [(1, 3000, None), (3, 1500, 1024), (64, 300, 128), (2, 40, 64)])
def test_tiled_score_mixing_decode_splits_its_keys(dev, batch, context, window):
    """Single tokens with long contexts: the keys of a token are split over CTAs and joined with the sink."""
    from einf_b200 import ops

    heads, kv_heads, size, page_size = 6, 2, 32, 16
    requests = [(context - 1 - 7 * (r % 5), 1) for r in range(batch)]
    (q, k, v, table, seq, pos), scale, window = _attention_case(dev, torch.bfloat16, heads, kv_heads, size, page_size,
                                                                requests, window)
    generator = torch.Generator().manual_seed(9)
    slopes, talk, sink = _mixing(heads, generator, dev)
    assert ops.mixed_tiled_splits(batch, 1, window, context) > 1 or context < 128
    out, want = torch.empty_like(q), torch.empty_like(q).cpu()
    st = status(dev)
    ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, window, slopes, talk, sink, 1.0, st,
                              q_tiles=torch.zeros((0, 4), dtype=torch.int32, device=dev), single_tokens=None,
                              num_singles=batch, max_context=context)
    ref.paged_attention_mixed(q.cpu(), k.cpu(), v.cpu(), table.cpu(), seq.cpu(), pos.cpu(), want, scale, window,
                              slopes.cpu(), talk.cpu(), sink.cpu(), 1.0, st.cpu())
    assert int(st) == 0
    torch.testing.assert_close(out.cpu(), want, **tol(torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tiled_score_mixing_far_key_and_window_edge(dev, dtype):
    """One key far back carries the weight: a query whose window still holds it returns its value, the next
    query, for which it has just left the window, does not; in a prompt portion and for a single token."""
    from einf_b200 import ops

    heads, kv_heads, size, page_size, window = 4, 2, 32, 16, 100
    needle = 37
    for requests in ([(0, 300)], [(needle + window - 1, 1), (needle + window, 1)], [(100, 60)]):
        (q, k, v, table, seq, pos), scale, _ = _attention_case(dev, dtype, heads, kv_heads, size, page_size,
                                                               requests, window)
        q[:] = 0.0
        q[:, :, 0] = 1.0
        k[:] = 0.0
        for r in range(len(requests)):
            page, offset = int(table[r, needle // page_size]), needle % page_size
            k[page, :, offset, 0] = 40.0 / scale
            v[page, :, offset, :] = 7.0
        out = torch.empty_like(q)
        st = status(dev)
        q_tiles, singles = _step_split(requests)
        ops.paged_attention_mixed(q, k, v, table, seq, pos, out, scale, window, None, None, None, 1.0, st,
                                  q_tiles=q_tiles.to(dev), single_tokens=singles.to(dev), num_singles=singles.shape[0],
                                  max_context=max(s + n for s, n in requests))
        assert int(st) == 0
        for t in range(q.shape[0]):
            p = int(pos[t])
            inside = needle <= p < needle + window
            got = out[t].abs().max().item()
            assert (abs(got - 7.0) < 1e-3) if inside else got < 6.0, (dtype, requests, p, got)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths", [(1, 1, 1), (5, 1, 33), (700,), (16, 17, 130, 2), (2100, 3)])
def test_gated_scan_in_segments(dev, dtype, lengths):
    from einf_b200 import ops

    blocks, part = 3, 20
    width = blocks * part
    tokens = sum(lengths)
    generator = torch.Generator().manual_seed(len(lengths) + tokens)
    gates = torch.randn((tokens, blocks, 2 * part), generator=generator)
    gate_bias = torch.randn((blocks, 2 * part), generator=generator)
    u = torch.randn((tokens, width), generator=generator).to(dtype)
    y_raw = torch.randn((tokens, width), generator=generator).to(dtype)
    y_bias = torch.randn((width,), generator=generator)
    rate = -8.0 * torch.nn.functional.softplus(torch.randn((width,), generator=generator) - 3.0)
    state = torch.randn((len(lengths) + 2, width), generator=generator)
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    q_start = torch.tensor(starts, dtype=torch.int32)
    slots = torch.tensor([(r + 1) % (len(lengths) + 2) for r in range(len(lengths))], dtype=torch.int32)
    want, want_state = torch.empty((tokens, width), dtype=dtype), state.clone()
    ref.gated_scan(gates, gate_bias, u, y_raw, y_bias, rate, want_state, q_start, slots, want, 1.3)
    got, got_state = torch.empty((tokens, width), dtype=dtype, device=dev), state.clone().to(dev)
    ops.gated_scan(gates.to(dev), gate_bias.to(dev), u.to(dev), y_raw.to(dev), y_bias.to(dev), rate.to(dev), got_state,
                   q_start.to(dev), slots.to(dev), got, 1.3, max_q_len=max(lengths))
    close = dict(rtol=2e-4, atol=2e-5) if dtype == torch.float32 else tol(dtype)
    torch.testing.assert_close(got.cpu(), want, **close)
    torch.testing.assert_close(got_state.cpu(), want_state, rtol=2e-4, atol=2e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens, hidden, side, layers_done", [
    (1, 64, 8, 0), (5, 72, 6, 2), (9, 100, 16, 1), (1030, 128, 64, 3), (8, 896, 64, 7), (3, 1544, 33, 0),
])
@pytest.mark.parametrize("parts", ["both", "token input", "depth average", "neither"])
def test_end_of_a_layer(dev, dtype, tokens, hidden, side, layers_done, parts):
    """The kernel that takes several tokens a CTA (widths that are multiples of eight) and the one that
    takes a row a CTA (the others): pending sublayer output, token input, depth average."""
    from einf_b200 import ops

    if parts != "both" and tokens not in (5, 1030):
        pytest.skip("the parts alone at two sizes")
    generator = torch.Generator().manual_seed(tokens + hidden)
    vocab = 50
    residual = torch.randn((tokens, hidden), generator=generator)
    pending = [torch.randn((tokens, hidden), generator=generator).to(dtype)]
    ids = torch.randint(0, vocab, (tokens,), generator=generator, dtype=torch.int32)
    table = torch.randn((vocab, side), generator=generator).to(dtype)
    gate = (torch.randn((side, hidden), generator=generator) * hidden ** -0.5).to(dtype)
    proj_t = torch.randn((side, hidden), generator=generator).to(dtype)
    norm = torch.rand((hidden,), generator=generator) + 0.5
    history = torch.randn((layers_done + 2, tokens, hidden), generator=generator)
    weight = torch.randn((layers_done + 2,), generator=generator)
    use_side, use_depth = parts in ("both", "token input"), parts in ("both", "depth average")

    def arguments(move):
        return (move(residual.clone()), [move(t) for t in pending], 0.6, move(ids),
                (move(table), move(gate), move(proj_t), move(norm), 1e-5) if use_side else None,
                (move(history.clone()), layers_done, move(weight)) if use_depth else None)

    want, got = arguments(lambda t: t), arguments(lambda t: t.to(dev))
    ref.stream_tail(*want)
    ops.stream_tail(*got)
    close = dict(rtol=2e-4, atol=2e-4) if dtype == torch.float32 else dict(rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(got[0].cpu(), want[0], **close)
    if use_depth:
        torch.testing.assert_close(got[5][0].cpu(), want[5][0], **close)


@pytest.mark.parametrize("tokens, hidden, side, layers_done, splits", [
    (150, 16, 16, 0, 1), (300, 896, 64, 3, 1), (149, 144, 32, 9, 3), (2401, 48, 48, 1, 1), (593, 1568, 64, 0, 2),
])
def test_end_of_a_layer_on_the_tensor_cores(dev, tokens, hidden, side, layers_done, splits):
    """Two to 16 tokens a CTA, widths around the warps' shares, partial sums: off the statement in 64 bits by what its 32-bit
    sums and norms round, 2^-24 of each of their terms."""
    from einf_b200 import ops

    generator = torch.Generator().manual_seed(tokens + side)
    vocab = 50
    residual = torch.randn((tokens, hidden), generator=generator)
    pending = [torch.randn((splits, tokens, hidden), generator=generator),
               torch.randn((tokens, hidden), generator=generator).to(torch.bfloat16)][:1 + splits % 2]
    ids = torch.randint(0, vocab, (tokens,), generator=generator, dtype=torch.int32)
    table, proj_t = (torch.randn((n, m), generator=generator).to(torch.bfloat16) for n, m in ((vocab, side), (side, hidden)))
    gate = (torch.randn((side, hidden), generator=generator) * hidden ** -0.5).to(torch.bfloat16)
    norm = torch.rand((hidden,), generator=generator) + 0.5
    history = torch.randn((layers_done + 2, tokens, hidden), generator=generator)
    weight = torch.randn((layers_done + 2,), generator=generator)
    x = residual.double() + 0.6 * sum(p.double().reshape(-1, tokens, hidden).sum(0) for p in pending)
    s = x @ gate.double().T
    g = 0.5 * s * (1 + torch.tanh(0.7978845608028654 * (s + 0.044715 * s ** 3))) * table[ids.long()].double()
    y = g @ proj_t.double()
    x = x + 0.6 * y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * norm.double()
    for depth in (True, False):
        got, line = residual.to(dev), history.to(dev)
        ops.stream_tail(got, [p.to(dev) for p in pending], 0.6, ids.to(dev),
                        (table.to(dev), gate.to(dev), proj_t.to(dev), norm.to(dev), 1e-5),
                        (line, layers_done, weight.to(dev)) if depth else None)
        want = x
        if depth:
            torch.testing.assert_close(line[layers_done + 1].cpu().double(), x, rtol=1e-5, atol=1e-5)
            want = weight[layers_done + 1].double() * x + torch.einsum("j,jth->th", weight[:layers_done + 1].double(),
                                                                      history[:layers_done + 1].double())
        torch.testing.assert_close(got.cpu().double(), want, rtol=1e-5, atol=2e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden, taps, lengths", [
    (64, 4, (1, 190, 2, 69)), (516, 2, (8, 8, 264, 3)), (1540, 3, (300,)), (2052, 4, (130, 1)), (72, 5, (66, 2)), (70, 3, (80,)),
    (2004, 4, (1, 190, 2, 69)), (1856, 2, (8, 8, 264, 3)), (4100, 3, (130, 1)),      # above 2^19 elements
    (2004, 4, (262,)), (1856, 2, (283,)), (4100, 3, (131,)),                          # one request
    (64, 4, (1, 1, 1)), (516, 2, (1, 1)), (896, 3, (1, 1, 1, 1)), (2052, 4, (1,)), (72, 5, (1, 1)),
])
def test_norm_and_convolution(dev, dtype, hidden, taps, lengths):
    """Rows in registers and runs of eight tokens (widths in groups of four, up to four taps), the kernels for the other
    widths and taps, and single tokens, whose launch moves the state on as well."""
    from einf_b200 import ops

    generator = torch.Generator().manual_seed(hidden + taps)
    tokens = sum(lengths)
    starts = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32)
    seq = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).to(torch.int32)
    slots = torch.tensor([2, 0, -1, 3], dtype=torch.int32)[:len(lengths)]
    residual = torch.randn((tokens, hidden), generator=generator)
    pending = [torch.randn((tokens, hidden), generator=generator).to(dtype),
               torch.randn((3, tokens, hidden), generator=generator)][:1 + taps % 2]
    weight = torch.rand((hidden,), generator=generator) + 0.5
    conv = torch.randn((hidden, taps), generator=generator)
    state = torch.randn((5, taps - 1, hidden), generator=generator)
    single = max(lengths) == 1

    def run(module, move):
        row, line, out = move(residual.clone()), move(state.clone()), move(torch.empty((tokens, hidden), dtype=dtype))
        module.norm_conv([move(t) for t in pending], 0.7, row, move(weight), 1e-5, move(conv), line, move(seq), move(starts),
                         move(slots), out, single_tokens=single)
        return row.cpu(), line.cpu(), out.cpu()

    for got, want in zip(run(ops, lambda t: t.to(dev)), run(ref, lambda t: t)):
        close = dict(rtol=1e-4, atol=2e-5) if got.dtype == torch.float32 else tol(dtype)
        torch.testing.assert_close(got, want, **close)
