"""The kernels behind the Tepavik mixers, each alone against its plain statement
(``kernel_references``): activations, unit-norm heads with the cache write, the
chunked and soft-capped attention (general kernel and the tcgen05 kernels), the
short convolution with its carried inputs, the recurrence with its state slots,
the gated norm.
"""
from __future__ import annotations

import random

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
@pytest.mark.parametrize("kind", ["relu2", "gelu_tanh", "silu", "relu"])
def test_activation(dev, dtype, kind):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(1)
    for shape in ((3, 37), (65, 256), (4, 3, 40)):        # the last: split-K partial sums
        x = (torch.randn(shape, generator=gen) * 2).to(torch.float32 if len(shape) == 3 else dtype).to(dev)
        out = torch.empty(shape[-2:], dtype=dtype, device=dev)
        want = torch.empty_like(out)
        ops.activation(x, out, kind)
        ref.activation(x, want, kind)
        close(out, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, key, value, eps", [
    (4, 2, 16, 24, 1e-5), (3, 1, 64, 64, None), (5, 5, 40, 8, 1e-6), (2, 0, 128, 128, 1e-5), (1, 1, 256, 200, 1e-5),
])
def test_qkv_norm_store(dev, dtype, heads, kv_heads, key, value, eps):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(2)
    tokens, page, pages = 11, 4, 9
    width = (heads + kv_heads) * key + kv_heads * value
    for splits in (1, 3):
        shape = (tokens, width) if splits == 1 else (splits, tokens, width)
        qkv = torch.randn(shape, generator=gen).to(dtype if splits == 1 else torch.float32).to(dev)
        bias = torch.randn(width, generator=gen).to(dev)
        slots = torch.randperm(page * pages, generator=gen)[:tokens].to(torch.int32)
        slots[3] = -1
        slots = slots.to(dev)
        outs = []
        for fn in (ops.qkv_norm_store, ref.qkv_norm_store):
            q = torch.zeros((tokens, heads, key), dtype=dtype, device=dev)
            k = torch.zeros((pages, max(kv_heads, 1), page, key), dtype=dtype, device=dev)
            v = torch.zeros((pages, max(kv_heads, 1), page, value), dtype=dtype, device=dev)
            st = status(dev)
            fn(qkv, bias, slots if kv_heads else None, q, k if kv_heads else None, v if kv_heads else None, heads,
               kv_heads, key, value, eps, st)
            assert int(st) == 0
            outs.append((q, k, v))
        for got, want in zip(*outs):
            close(got, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, size, value, page_size, chunk, softcap", [
    (4, 2, 16, 24, 4, 7, 5.0), (3, 1, 32, 8, 8, 1, None), (6, 2, 64, 64, 16, 50, 30.0), (2, 2, 20, 36, 16, 16, 2.0),
    (7, 1, 128, 256, 8, 33, None),
])
def test_general_attention_with_chunks_caps_and_value_sizes(dev, dtype, heads, kv_heads, size, value, page_size, chunk,
                                                            softcap):
    from einf_b200 import ops

    requests = [(0, 1), (0, 2 * page_size), (chunk - 1, 3), (3 * chunk - 2, 5), (chunk * 4, 1), (chunk * 4 - 1, 1),
                (70, 1), (0, 37)]
    (q, k, v, table, seq, pos), scale, _ = _attention_case(dev, dtype, heads, kv_heads, size, page_size, requests, None)
    v = torch.randn((k.shape[0], kv_heads, page_size, value), generator=torch.Generator().manual_seed(3)).to(dtype).to(dev)
    out = torch.empty((q.shape[0], heads, value), dtype=dtype, device=dev)
    want = torch.empty_like(out)
    st = status(dev)
    ops.paged_attention_generic(q, k, v, table, seq, pos, out, scale * 3, None, st, chunk=chunk, softcap=softcap)
    ref.paged_attention_generic(q, k, v, table, seq, pos, want, scale * 3, None, st, chunk=chunk, softcap=softcap)
    assert int(st) == 0
    close(out, want, dtype)


@pytest.mark.parametrize("first_case", [0, 12])
def test_tcgen05_attention_with_chunks_and_caps(dev, first_case):
    """Seeded random launches of the tcgen05 prefill and decode kernels with a chunked mask and a
    soft cap: chunk sizes that are no multiple of a page or a tile, portions that start and end
    anywhere (just inside and just outside a chunk's edge among them), single tokens at a chunk's
    first and last position, keys scaled so that the cap bites; against the general kernel."""
    from einf_b200 import ops

    for case in range(first_case, first_case + 12):
        rng = random.Random(1000 + case)
        size, page_size = rng.choice([64, 128]), rng.choice([8, 16, 32, 64, 128])
        kv_heads, group = rng.choice([1, 2, 4]), rng.choice([1, 2, 3, 8])
        chunk = rng.choice([1, 5, 50, 128, 200, 777, 1024, None])
        softcap = rng.choice([None, 2.0, 20.0, 50.0])
        window = rng.choice([None, None, None, 90])
        edge = chunk or 100
        requests = []
        for _ in range(rng.randint(1, 4)):
            start = rng.choice([0, edge - 1, edge, 3 * edge - 2, rng.randrange(1, 200), rng.randrange(200, 2500)])
            requests.append((start, rng.choice([2, 3, edge + 1, rng.randrange(2, 140), rng.randrange(100, 600)])))
        singles = [(rng.choice([edge - 1, edge, 2 * edge + 1, 4 * edge - 1, rng.randrange(1, 3000)]), 1)
                   for _ in range(rng.randint(1, 5))]
        layout = rng.choice(["shuffled", "runs"])
        heads = kv_heads * group
        (q, k, v, table, seq, pos), scale, _ = _attention_case(dev, torch.bfloat16, heads, kv_heads, size, page_size,
                                                               requests + singles, window, seed=case, layout=layout)
        k.mul_(rng.choice([1.0, 3.0, 8.0]))
        tiles, cursor = [], 0
        for r, (start, q_len) in enumerate(requests):
            for first in range(0, q_len, ops.Q_TILE):
                tiles.append((r, cursor + first, min(ops.Q_TILE, q_len - first), start + first))
            cursor += q_len
        q_tiles = torch.tensor(tiles, dtype=torch.int32, device=dev)
        single_tokens = torch.arange(cursor, cursor + len(singles), dtype=torch.int32, device=dev)
        st = status(dev)
        want = torch.empty_like(q)
        ops.paged_attention_generic(q, k, v, table, seq, pos, want, scale, window, st, chunk=chunk, softcap=softcap)
        out = torch.full_like(q, float("nan"))
        ops.paged_prefill_attention(q, k, v, table, q_tiles, out, scale, window, st, use_tcgen05=True,
                                    prefill_cluster=rng.randrange(0, 5), cached_before=max(s for s, _ in requests),
                                    chunk=chunk, softcap=softcap)
        ops.paged_decode_attention_tcgen05(q, k, v, table, seq, pos, out, scale, window, rng.choice([1, 2, 4, 8]), st,
                                           single_tokens, chunk=chunk, softcap=softcap)
        assert int(st) == 0, case
        torch.testing.assert_close(out, want, **tol(torch.bfloat16), msg=lambda m: f"case {case}: {m}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, size, value_size, page, options", [
    (2, 1, 64, 64, 16, {}), (3, 3, 128, 128, 8, {"window": 50}), (2, 2, 4, 68, 16, {"window": 40, "keep_first": 70}),
    (4, 2, 36, 20, 64, {"chunk": 48, "softcap": 4.0}), (2, 1, 96, 64, 16, {"in_keys": True, "sink": True, "gate": True}),
    (2, 1, 64, 100, 16, {"sink": True, "value_gate": True, "window": 64}),
])
@pytest.mark.parametrize("requests", [[(0, 8)], [(0, 33), (70, 1), (61, 67)], [(5, 129), (0, 32), (0, 1)]])
def test_attention_of_portions_shares_keys(dev, dtype, heads, kv_heads, size, value_size, page, options, requests):
    """Portions of prompts through the kernel that reads a key row once for 32 tokens, single tokens beside them,
    against the plain statement: rows around its tiles of 32 tokens and 64 keys, every option of the general kernel."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(size + value_size + len(requests))
    options = dict(options)
    window, in_keys = options.pop("window", None), options.pop("in_keys", False)
    tokens = sum(n for _, n in requests)
    if options.pop("sink", False):
        options["sink"] = torch.randn(heads, generator=gen).to(dev)
    if options.pop("gate", False):
        options["gate"] = torch.rand((tokens, heads), generator=gen).to(dev)
    if options.pop("value_gate", False):
        options["value_gate"] = torch.randn((tokens, heads * value_size), generator=gen).to(dtype).to(dev)
    pages = [-(-(start + n) // page) for start, n in requests]
    order = torch.randperm(sum(pages), generator=gen).to(torch.int32)
    table = torch.full((len(requests), max(pages)), -1, dtype=torch.int32)
    seq, pos, tiles, singles = [], [], [], []
    for r, ((start, n), own) in enumerate(zip(requests, torch.split(order, pages))):
        table[r, :own.shape[0]] = own
        if n == 1:
            singles.append(len(seq))
        else:
            tiles += [(r, len(seq) + first, min(128, n - first), start + first) for first in range(0, n, 128)]
        seq, pos = seq + [r] * n, pos + list(range(start, start + n))
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=dev)  # noqa: E731
    q = torch.randn((tokens, heads, size), generator=gen).to(dtype).to(dev)
    k = torch.randn((sum(pages), kv_heads, page, size), generator=gen).to(dtype).to(dev)
    v = None if in_keys else torch.randn((sum(pages), kv_heads, page, value_size), generator=gen).to(dtype).to(dev)
    if in_keys:
        options["values_in_keys"] = value_size
    st = status(dev)
    out, want = (torch.full((tokens, heads, value_size), float("nan"), dtype=dtype, device=dev) for _ in range(2))
    assert ops._takes_prompt_tiles(ints(tiles).view(-1, 4), tokens - len(singles), size, value_size,
                                   size if in_keys else value_size, k, k if in_keys else v)
    before = ops.launch_count
    ops.paged_attention_generic(q, k, v, table.to(dev), ints(seq), ints(pos), out, size ** -0.5, window, st,
                                q_tiles=ints(tiles).view(-1, 4), single_tokens=ints(singles), **options)
    assert ops.launch_count - before == 1 + bool(singles)
    ref.paged_attention_generic(q, k, v, table.to(dev), ints(seq), ints(pos), want, size ** -0.5, window, st, **options)
    assert int(st) == 0
    close(out, want, dtype)


def _packed(lengths, dev):
    starts = [0]
    seq = []
    for r, n in enumerate(lengths):
        starts.append(starts[-1] + n)
        seq += [r] * n
    return (torch.tensor(starts, dtype=torch.int32, device=dev), torch.tensor(seq, dtype=torch.int32, device=dev))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("channels, taps, heads", [(24, 4, 3), (40, 2, 0), (7, 5, 2), (64, 1, 1), (130, 16, 4)])
def test_conv_silu_carries_its_inputs(dev, dtype, channels, taps, heads):
    """Portions of 1, 2 and many tokens (shorter and longer than the kernel), a request without a
    slot, slots in any order, two steps in a row on the same states."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(4)
    slots = torch.tensor([2, -1, 0, 3, 1], dtype=torch.int32, device=dev)
    states = [torch.randn((5, 9 + (taps - 1) * channels), generator=gen).to(dev) for _ in range(1)] * 1
    state_got, state_want = states[0].clone(), states[0].clone()
    for lengths in ((1, 2, 9, 1, taps), (3, 1, 1, 2 * taps + 1, 2)):
        q_start, seq = _packed(lengths, dev)
        tokens = sum(lengths)
        wide = torch.randn((tokens, 5 + channels + heads), generator=gen).to(dtype).to(dev)
        x, dt_raw = wide[:, 5:5 + channels], wide[:, 5 + channels:]
        weight = torch.randn((channels, taps), generator=gen).to(dev)
        bias = torch.randn(channels, generator=gen).to(dev)
        dt_bias, a_log = torch.randn(heads, generator=gen).to(dev), torch.randn(heads, generator=gen).to(dev)
        results = []
        for fn, state in ((ops.conv_silu, state_got), (ref.conv_silu, state_want)):
            out = torch.empty((tokens, channels), dtype=dtype, device=dev)
            dt, decay = torch.empty((tokens, heads), device=dev), torch.empty((tokens, heads), device=dev)
            view = state[:, 9:].view(5, taps - 1, channels)
            if heads:
                fn(x, weight, bias, view, seq, q_start, slots, out, dt_raw, dt_bias, a_log, dt, decay)
            else:
                fn(x, weight, bias, view, seq, q_start, slots, out)
            results.append((out, dt, decay) if heads else (out,))
        for got, want in zip(*results):
            close(got, want, dtype)
        torch.testing.assert_close(state_got, state_want, rtol=0, atol=0)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, groups, dim, vdim, per_token, silu", [
    (3, 3, 24, 16, False, True), (4, 2, 8, 12, True, False), (2, 1, 128, 64, True, False), (1, 1, 40, 8, False, True),
    (6, 3, 20, 8, True, False), (2, 2, 16, 130, False, False), (8, 8, 64, 64, False, True), (2, 1, 300, 20, True, False),
])
@pytest.mark.parametrize("rows, segment_len, columns", [(0, None, 0), (4, 3, 1), (8, None, 1), (16, 16, 2), (0, 5, 0),
                                                        (16, None, 2)])
def test_linear_recurrence_keeps_its_state(dev, dtype, heads, groups, dim, vdim, per_token, silu, rows, segment_len,
                                           columns):
    """Two steps on the same slots (one request without a slot), portions of one token and of many,
    an empty request; inputs as columns of a wider matrix; every number of rows per thread; portions
    cut into segments that run side by side; outputs and states against the plain loop."""
    if rows and 32 * rows < dim:
        pytest.skip("too few rows per thread for this state")
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(5)
    slots = torch.tensor([1, -1, 3, 0], dtype=torch.int32, device=dev)
    base = torch.randn((4, 5 + heads * dim * vdim), generator=gen).to(dev)
    state_got, state_want = base.clone(), base.clone()
    for lengths in ((1, 3, 17, 0), (40, 1, 1, 2), (1, 1, 1, 1)):     # the last: a step of single tokens
        q_start, _ = _packed(lengths, dev)
        tokens = sum(lengths)
        wide = (torch.randn((tokens, 8 + 2 * groups * dim + heads * vdim), generator=gen) * 0.5).to(dtype).to(dev)
        q, k = wide[:, 8:8 + groups * dim], wide[:, 8 + groups * dim:8 + 2 * groups * dim]
        v = wide[:, 8 + 2 * groups * dim:]
        kwargs = dict(silu_inputs=silu)
        if per_token:
            kwargs.update(token_decay=torch.rand((tokens, heads), generator=gen).to(dev),
                          token_scale=torch.rand((tokens, heads), generator=gen).to(dev),
                          skip=torch.randn(heads, generator=gen).to(dev))
        else:
            kwargs.update(head_decay=torch.rand(heads, generator=gen).to(dev))
        ys = []
        for fn, state in ((ops.linear_recurrence, state_got), (ref.linear_recurrence, state_want)):
            y = torch.zeros((tokens, heads * vdim), device=dev)
            fn(q, k, v, state[:, 5:].view(4, heads, dim, vdim), q_start, slots, y, heads, groups, dim, vdim,
               max_q_len=max(lengths), rows=rows, segment_len=segment_len, columns=columns, **kwargs)
            ys.append(y)
        torch.testing.assert_close(ys[0], ys[1], rtol=2e-4, atol=2e-4)
        torch.testing.assert_close(state_got, state_want, rtol=2e-4, atol=2e-4)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("options", [{}, {"window": 37}, {"window": 20, "keep_first": 9}, {"chunk": 48}])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_attention_of_portions_keeps_a_value_from_rows_that_do_not_see_it(dev, dtype, options, bad):
    """A value that is not finite reaches the tokens that see its key and no other: those before it, those whose window has
    passed it and those of the next chunk are bit for bit what they are beside a finite one."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(5)
    start, tokens, heads, size, page = 30, 100, 2, 32, 16
    options = dict(options)
    window, keep, chunk = options.pop("window", None), options.get("keep_first", 0), options.get("chunk")
    pages = -(-(start + tokens) // page)
    table = torch.randperm(pages, generator=gen).to(torch.int32).view(1, -1).to(dev)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=dev)  # noqa: E731
    q, k, v = (torch.randn(shape, generator=gen).to(dtype).to(dev) for shape in (
        (tokens, heads, size), (pages, heads, page, size), (pages, heads, page, size)))
    tiles, none, st = ints([(0, 0, tokens, start)]), ints([]), status(dev)
    seq, pos = ints([0] * tokens), ints(range(start, start + tokens))

    def run(values):
        out = torch.empty((tokens, heads, size), dtype=dtype, device=dev)
        ops.paged_attention_generic(q, k, values, table, seq, pos, out, size ** -0.5, window, st, q_tiles=tiles,
                                    single_tokens=none, **options)
        return out

    clean = run(v)
    assert bool(torch.isfinite(clean).all()) and int(st) == 0
    for key in (5, 31, 64, 95, 129):
        broken = v.clone()
        broken[int(table[0, key // page]), :, key % page] = bad
        got, at = run(broken), pos.long()
        sees = (at >= key) & ((at < key + window) | (key < keep) if window else at >= 0)
        if chunk:
            sees &= at // chunk == key // chunk
        assert not bool(torch.isfinite(got[sees]).any()) and torch.equal(got[~sees], clean[~sees]), key


@pytest.mark.parametrize("heads, groups, dim, vdim, per_token, silu, pad", [
    (2, 2, 64, 64, False, True, 8), (4, 1, 128, 64, True, False, 8), (1, 1, 128, 260, True, False, 4), (3, 3, 64, 132, True, True, 4),
    (2, 2, 16, 12, True, False, 4), (2, 1, 40, 100, False, False, 8), (1, 1, 100, 36, False, True, 4),
])
@pytest.mark.parametrize("lengths, segment_len", [
    ((24,), None), ((63, 1), None), ((64, 0, 65), None), ((130, 16, 1, 193), None), ((130, 16, 1, 193), 128), ((250,), 256),
])
def test_chunked_recurrence(dev, heads, groups, dim, vdim, per_token, silu, pad, lengths, segment_len):
    """The chunked form against the plain loop in 64 bits: portions around its tiles of 16, chunks of 64 and
    segments, single tokens and an empty request beside them, a request without a slot, decays that are zero, columns of
    wider matrices on 8- and 16-byte borders, states that fill no tile.  The bound: what both add up are the same products,
    so an element is off by at most (roundings on its way) x 2^-24 x (the sum of its products' sizes, which the loop on the
    absolute values gives); a product passes at most 16 rounded sums of 16 in each of two chains, eight roundings of its
    weight and one per segment."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim + vdim + sum(lengths))
    requests = len(lengths)
    slots = torch.arange(requests, dtype=torch.int32, device=dev)
    if requests > 2:
        slots[2] = -1
    base = torch.randn((requests, 4 + heads * dim * vdim), generator=gen).to(dev)
    q_start, _ = _packed(lengths, dev)
    tokens = sum(lengths)
    wide = (torch.randn((tokens, pad + 2 * groups * dim + heads * vdim + 12), generator=gen) * 0.5).to(torch.bfloat16).to(dev)
    q, k = wide[:, pad:pad + groups * dim], wide[:, pad + groups * dim:pad + 2 * groups * dim]
    v = wide[:, pad + 2 * groups * dim:pad + 2 * groups * dim + heads * vdim]
    kwargs = dict(silu_inputs=silu)
    if per_token:
        decay = torch.rand((tokens, heads), generator=gen)
        decay[torch.rand((tokens, heads), generator=gen) < 0.05] = 0.0
        kwargs.update(token_decay=decay.to(dev), token_scale=torch.rand((tokens, heads), generator=gen).to(dev),
                      skip=torch.randn(heads, generator=gen).to(dev))
    else:
        kwargs.update(head_decay=(1.0 - 0.1 * torch.rand(heads, generator=gen)).to(dev))
    state = base.clone()
    y = torch.full((tokens, heads * vdim), float("nan"), device=dev)
    view = state[:, 4:].view(requests, heads, dim, vdim)
    assert ops.recurrence_takes_chunks(q, k, v, view, y, dim, vdim, max(lengths)) == (max(lengths) >= ops.RECURRENCE_CHUNK_MIN)
    ops.linear_recurrence(q, k, v, view, q_start, slots, y, heads, groups, dim, vdim, max_q_len=max(lengths),
                          segment_len=segment_len, chunks=True, **kwargs)
    want = _recurrence64(q, k, v, base[:, 4:].view(requests, heads, dim, vdim), q_start, slots, heads, groups, lambda t: t, **kwargs)
    size = _recurrence64(q, k, v, base[:, 4:].view(requests, heads, dim, vdim), q_start, slots, heads, groups, torch.abs, **kwargs)
    bound = (32 + 8 + max(lengths) / 64) * 2.0 ** -24
    for got, exact, most in zip((y, view), want, size):
        assert bool(((got.double() - exact).abs() <= bound * most.abs() + 1e-12).all())
    if requests > 1:
        assert torch.equal(state[:, :4], base[:, :4])


@pytest.mark.parametrize("known", [False, True])
@pytest.mark.parametrize("dim, vdim, silu", [(64, 64, True), (128, 260, False), (40, 20, True), (16, 516, False)])
@pytest.mark.parametrize("lengths", [
    (130,) + (1,) * 40, (1, 24, 0, 193, 1, 64), (23, 24, 2, 65, 1, 0), (300, 17, 1) * 15, (1,) * 33 + (70,), (64, 64, 64)])
def test_a_portions_recurrence_goes_by_its_own_length(dev, dim, vdim, silu, lengths, known):
    """Every portion of a step gives bit for bit what it gives alone: those of 24 tokens and more through the chunked kernel,
    the others token by token, whatever stands beside them and whether the host knows the lengths."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim + vdim)
    heads, requests, tokens = 2, len(lengths), sum(lengths)
    q_start, _ = _packed(lengths, dev)
    slots = torch.randperm(requests, generator=gen).to(torch.int32).to(dev)
    base = torch.randn((requests, heads, dim, vdim), generator=gen).to(dev)
    q, k, v = ((torch.randn((tokens, heads * n), generator=gen) * 0.3).to(torch.bfloat16).to(dev) for n in (dim, dim, vdim))
    decay = torch.rand((tokens, heads), generator=gen).add(0.1).to(dev)

    def run(first, last, q_start, slots, state, lens, **options):
        y = torch.full((last - first, heads * vdim), float("nan"), device=dev)
        ops.linear_recurrence(q[first:last], k[first:last], v[first:last], state, q_start, slots, y, heads, heads, dim, vdim,
                              token_decay=decay[first:last], silu_inputs=silu, max_q_len=max(lens), **options)
        return y

    state, alone = base.clone(), base.clone()
    y = run(0, tokens, q_start, slots, state, lengths, **(dict(q_lens=lengths) if known else {}))
    for r, n in enumerate(lengths):
        if n == 0:
            continue
        first = int(q_start[r])
        # a single token beside a prompt takes the streaming kernel only where the host knows of nothing but single tokens
        only_singles = known and not any(1 < m < 24 for m in lengths)
        options = {} if n >= 24 or (n == 1 and only_singles) else dict(segment_len=23)
        got = y[first:first + n]
        want = run(first, first + n, torch.tensor([0, n], dtype=torch.int32, device=dev), slots[r:r + 1], alone, [n], **options)
        assert torch.equal(got, want), (r, n)
    assert torch.equal(state, alone)


@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("dim, vdim", [(64, 64), (128, 20), (40, 132)])
@pytest.mark.parametrize("lengths", [(60,), (40, 150)])
@pytest.mark.parametrize("what", ["v", "k", "q", "scale", "decay"])
def test_chunked_recurrence_keeps_what_is_not_finite_from_earlier_tokens(dev, silu, dim, vdim, lengths, what):
    """An infinity in one token's inputs leaves the tokens before it, the other requests and, in a value, the other columns bit
    for bit as they were, and what it belongs to is no number afterwards (the token's own output with a query, everything
    from the token on and the state otherwise)."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(dim + vdim)
    heads, requests, tokens = 2, len(lengths), sum(lengths)
    q_start, _ = _packed(lengths, dev)
    slots = torch.arange(requests, dtype=torch.int32, device=dev)
    base = torch.randn((requests, heads, dim, vdim), generator=gen).to(dev)
    inputs = {name: torch.rand((tokens, heads * n), generator=gen).add(0.1).to(torch.bfloat16).to(dev)
              for name, n in (("q", dim), ("k", dim), ("v", vdim))}
    inputs["decay"], inputs["scale"] = (torch.rand((tokens, heads), generator=gen).add(0.1).to(dev) for _ in range(2))

    def run(with_inputs):
        state, y = base.clone(), torch.empty((tokens, heads * vdim), device=dev)
        ops.linear_recurrence(with_inputs["q"], with_inputs["k"], with_inputs["v"], state, q_start, slots, y, heads, heads, dim,
                              vdim, token_decay=with_inputs["decay"], token_scale=with_inputs["scale"], silu_inputs=silu,
                              max_q_len=max(lengths), chunks=True)
        return y.view(tokens, heads, vdim), state

    clean_y, clean_state = run(inputs)
    assert bool(torch.isfinite(clean_y).all()) and bool(torch.isfinite(clean_state).all())
    last_first = tokens - lengths[-1]                  # of the last request, which holds every token below
    for token in (last_first + 5, last_first + 31, tokens - 1):
        broken = {name: t.clone() for name, t in inputs.items()}
        head, column = 1, 3                            # the first head stays as it is
        width = {"q": dim, "k": dim, "v": vdim}.get(what, 1)
        broken[what][token, head * width + (column if width > 1 else 0)] = float("inf")
        y, state = run(broken)
        touched = torch.zeros_like(clean_y, dtype=torch.bool)
        end = token + 1 if what == "q" else tokens
        touched[token:end, head, column if what == "v" else slice(None)] = True
        assert torch.equal(y[~touched], clean_y[~touched]), (token, "reaches what it does not belong to")
        assert not bool(torch.isfinite(y[touched]).any()), (token, "is lost")
        of_state = torch.zeros_like(base, dtype=torch.bool)
        if what == "v":
            of_state[-1, head, :, column] = True
        elif what == "k":
            of_state[-1, head, column] = True
        elif what != "q":
            of_state[-1, head] = True
        assert torch.equal(state[~of_state], clean_state[~of_state]) and not bool(torch.isfinite(state[of_state]).any())


def _recurrence64(q, k, v, state, q_start, slots, heads, groups, of, head_decay=None, token_decay=None, token_scale=None,
                  skip=None, silu_inputs=False):
    """y and the states after the loop over tokens in 64 bits, of ``of`` the inputs (torch.abs: the sums of the sizes)."""
    tokens, dim, vdim = q.shape[0], state.shape[2], state.shape[3]
    q, k, v = (t.double() for t in (q, k, v))
    if silu_inputs:
        q, k, v = (t * torch.sigmoid(t) for t in (q, k, v))
    head_of = torch.arange(heads, device=q.device) // (heads // groups)
    q, k = (of(t).view(tokens, groups, dim)[:, head_of] for t in (q, k))
    v = of(v).view(tokens, heads, vdim)
    decay = token_decay.double() if head_decay is None else head_decay.double().expand(tokens, heads)
    scale = torch.ones_like(decay) if token_scale is None else token_scale.double()
    after, y = state.double().clone(), torch.zeros((tokens, heads, vdim), dtype=torch.float64, device=q.device)
    for r in range(slots.shape[0]):
        slot = int(slots[r])
        S = of(after[slot]) if slot >= 0 else torch.zeros_like(after[0])
        for t in range(int(q_start[r]), int(q_start[r + 1])):
            S = decay[t][:, None, None] * S + k[t][:, :, None] * (scale[t][:, None] * v[t])[:, None, :]
            y[t] = torch.einsum("hd,hdv->hv", q[t], S)
            if skip is not None:
                y[t] += of(skip.double())[:, None] * v[t]
        if slot >= 0 and q_start[r + 1] > q_start[r]:
            after[slot] = S
    return y.view(tokens, -1), after


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width, parts, gate_first, kind", [
    (48, 2, True, "silu"), (64, 1, False, "sigmoid"), (600, 3, True, "silu"), (40, 40, False, "silu"),
])
def test_gated_norm(dev, dtype, width, parts, gate_first, kind):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(6)
    tokens = 9
    y = torch.randn((tokens, width), generator=gen).to(dev)
    wide = torch.randn((tokens, width + 24), generator=gen).to(dtype).to(dev)
    gate = wide[:, 8:8 + width]
    weight = torch.randn(width, generator=gen).to(dev)
    out, want = (torch.empty((tokens, width), dtype=dtype, device=dev) for _ in range(2))
    ops.gated_norm(y, gate, weight, out, parts, 1e-5, gate_first, kind)
    ref.gated_norm(y, gate, weight, want, parts, 1e-5, gate_first, kind)
    close(out, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("channels, taps, heads, lengths", [
    (24, 4, 3, (1, 190, 2, 69)), (40, 2, 0, (8, 8, 264, 3)), (64, 1, 1, (65,)), (132, 3, 2, (3, 1, 191)),
    (2004, 4, 3, (1, 190, 2, 69)), (1856, 2, 0, (8, 8, 264, 3)), (8068, 1, 1, (65,)), (2692, 3, 2, (3, 1, 191)),    # 2^19 elements
    (2004, 4, 3, (262,)), (1856, 2, 0, (283,)), (2692, 3, 2, (195,)),     # one request: the same launch moves its state on
])
def test_conv_silu_over_runs_of_tokens(dev, dtype, channels, taps, heads, lengths):
    """Portions of 64 tokens and more on average, from 2^19 elements on four channels of eight tokens a thread: requests that
    begin inside a run, a request without a slot, a last run that is not full; and the same just below, an element a thread."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(8)
    slots = torch.tensor([2, 0, -1, 3], dtype=torch.int32, device=dev)[:len(lengths)]
    q_start, seq = _packed(lengths, dev)
    tokens = sum(lengths)
    wide = torch.randn((tokens, 4 + channels + 4), generator=gen).to(dtype).to(dev)
    x, dt_raw = wide[:, 4:4 + channels], wide[:, 4 + channels:4 + channels + heads]
    weight, bias = torch.randn((channels, taps), generator=gen).to(dev), torch.randn(channels, generator=gen).to(dev)
    dt_bias, a_log = torch.randn(heads, generator=gen).to(dev), torch.randn(heads, generator=gen).to(dev)
    state = torch.randn((5, 9 + (taps - 1) * channels), generator=gen).to(dev)
    results = []
    for fn in (ops.conv_silu, ref.conv_silu):
        out = torch.empty((tokens, channels), dtype=dtype, device=dev)
        dt, decay = torch.empty((tokens, heads), device=dev), torch.empty((tokens, heads), device=dev)
        mine = state.clone()
        extra = (dt_raw, dt_bias, a_log, dt, decay) if heads else (None,) * 5
        fn(x, weight, bias, mine[:, 9:].view(5, taps - 1, channels), seq, q_start, slots, out, *extra, activation=taps != 3,
           input_bias=bias if taps == 2 else None)
        results.append((out, dt, decay, mine) if heads else (out, mine))
    for got, want in zip(*results):
        close(got, want, dtype if got.dtype == dtype else torch.float32)


@pytest.mark.parametrize("which", ["conv_silu", "norm_conv"])
@pytest.mark.parametrize("end", [700, 693, 4, 2, 1])
def test_one_requests_state_ends_where_the_request_ends(dev, which, end):
    """Rows behind the end of a step's only request (its tokens moved over runs of eight) are no inputs of its state; a
    portion shorter than the state keeps the tail of the old one."""
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(end)
    tokens, channels, taps = 701, 900, 4
    x, weight = torch.randn((tokens, channels), generator=gen).to(dev), torch.randn((channels, taps), generator=gen).to(dev)
    state = torch.randn((3, taps - 1, channels), generator=gen).to(dev)
    q_start, slots = torch.tensor([0, end], dtype=torch.int32, device=dev), torch.tensor([1], dtype=torch.int32, device=dev)
    seq, results = torch.zeros(tokens, dtype=torch.int32, device=dev), []
    for module in (ops, ref):
        mine, out = state.clone(), torch.zeros((tokens, channels), device=dev)
        if which == "conv_silu":
            module.conv_silu(x, weight, None, mine, seq, q_start, slots, out)
        else:
            module.norm_conv([], 1.0, x.clone(), torch.ones(channels, device=dev), 1e-5, weight, mine, seq, q_start, slots, out)
        results.append((mine, out[:end]))
    for got, want in zip(*results):
        close(got, want, torch.float32)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width, parts, kind", [(252, 1, "silu"), (1280, 2, "sigmoid"), (1024, 1, "silu"), (1028, 1, "silu")])
def test_gated_norm_a_warp_a_row(dev, dtype, width, parts, kind):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(9)
    tokens = 593
    y = torch.randn((tokens, width), generator=gen).to(dev)
    gate = torch.randn((tokens, width + 24), generator=gen).to(dtype).to(dev)[:, 8:8 + width]
    weight = torch.randn(width, generator=gen).to(dev)
    for first in (True, False):
        out, want = (torch.empty((tokens, width), dtype=dtype, device=dev) for _ in range(2))
        ops.gated_norm(y, gate, weight, out, parts, 1e-5, first, kind)
        ref.gated_norm(y, gate, weight, want, parts, 1e-5, first, kind)
        close(out, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, vdim", [(3, 4), (2, 128), (1, 252), (2, 1024)])
def test_memory_output_four_elements_a_load(dev, dtype, heads, vdim):
    from einf_b200 import ops

    gen = torch.Generator().manual_seed(10)
    tokens, columns = 7, ops.memory_value_columns(vdim)
    y = torch.randn((tokens, heads * columns), generator=gen).to(dev)
    floor = torch.rand((tokens, heads), generator=gen).to(dev)
    gate = torch.randn((tokens, heads * vdim + 8), generator=gen).to(dtype).to(dev)[:, 4:4 + heads * vdim]
    weight = torch.randn(heads * vdim, generator=gen).to(dev)
    out, want = (torch.empty((tokens, heads * vdim), dtype=dtype, device=dev) for _ in range(2))
    for fn, to in ((ops.memory_output, out), (ref.memory_output, want)):
        fn(y, floor, gate, weight, to, heads, vdim, 0.125, 1e-5, 1e-6)
    close(out, want, dtype)
