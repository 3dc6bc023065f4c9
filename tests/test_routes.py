"""Which calls go which way, and what the host hands on, on a machine without a GPU."""
from dataclasses import replace

import pytest
import torch


def test_parts_of_ones_own_keep_their_forward():
    """Parts derived from the attention mixer and the gated feed-forward, under kinds of their own, run their own
    ``forward`` for any number of tokens; the built-in ones take the kernels for a few."""
    from conftest import SIZED
    from einf_b200.config import config_from_dict
    from einf_b200.parts import base
    from einf_b200.parts.attention import PagedAttention
    from einf_b200.parts.block import build_block
    from einf_b200.parts.mlp import GatedMLP
    from einf_b200.parts.model import expected_tensors
    from einf_b200.weights.random import random_tensors

    config = config_from_dict(dict(SIZED["0.5b"], vocab_size=64, num_hidden_layers=1))
    spec = config.model_spec()
    tensors = random_tensors(expected_tensors(spec)[0], 0)
    runtime, called = base.Runtime(torch.bfloat16, torch.device("cpu")), []

    class Mixer(PagedAttention):
        def forward(self, x, ctx, cache):
            called.append("mixer")
            return x

    class FeedForward(GatedMLP):
        def forward(self, x, ctx):
            called.append("feed_forward")
            return x

    saved = {category: dict(kinds) for category, kinds in base._REGISTRY.items()}
    try:
        base.register_part("mixer", "own_mixer")(Mixer)
        base.register_part("feed_forward", "own_feed_forward")(FeedForward)
        built_in = build_block(spec.layers[0], tensors, runtime)
        assert built_in.mixer.takes_few() and built_in.feed_forward.takes_few()
        for own in ({"mixer"}, {"feed_forward"}, {"mixer", "feed_forward"}):
            parts = {role: replace(part, kind="own_" + role) if role in own else part for role, part in spec.layers[0].parts.items()}
            block = build_block(replace(spec.layers[0], parts=parts), tensors, runtime)
            block.mixer_norm.forward = block.feed_forward_norm.forward = lambda pending, residual, **_: residual
            for role in {"mixer", "feed_forward"} - own:
                getattr(block, role).forward = lambda x, *_: x
            called.clear()
            block.forward(torch.zeros(4, 896), None, type("Context", (), {"status": None}), None)
            assert set(called) == own
    finally:
        for category, kinds in saved.items():
            base._REGISTRY[category].clear()
            base._REGISTRY[category].update(kinds)


@pytest.mark.parametrize("hidden, inter, limit", [(896, 4864, 16), (960, 5120, 16), (1024, 4608, 16), (1024, 4736, 16), (1024, 4768, 8), (992, 5120, 8)])
def test_more_than_eight_tokens_where_gate_up_is_one_wave(monkeypatch, hidden, inter, limit):
    from einf_b200 import ops

    monkeypatch.setattr(ops, "_sm_count", lambda: 148)
    ops.few_tokens_limit.cache_clear()
    assert ops.few_tokens_limit(hidden, inter) == limit
    ops.few_tokens_limit.cache_clear()


@pytest.mark.parametrize("rows", [65535 * 128, 65535 * 128 + 1])
def test_rows_of_a_32_bit_product_in_parts(rows):
    """As many tiles of 128 rows as the launcher takes (its grid's second dimension), not one row more."""
    from einf_b200 import ops

    x, weight, out = (torch.empty(size, device="meta") for size in ((rows, 8), (16, 8), (rows, 16)))
    assert ops.gemm_parts_takes(x, weight, out) == (rows <= 65535 * 128)


class _Others:
    """Sampling parameters of another type."""

    def __init__(self, params):
        for name in ("temperature", "top_p", "min_p", "top_k", "seed"):
            setattr(self, name, getattr(params, name))


@pytest.mark.parametrize("collection", ["list", "views", "others", "derived"])
def test_sampling_parameters_of_any_collection_and_type(monkeypatch, collection):
    """The step's staging holds the same for sequences of sampling parameters, for views of a dict, for other objects with
    their attributes, and for a derived class's own properties."""
    from einf_b200 import ops
    from einf_b200.cache.control import SamplingParams
    from einf_b200.sampling import Sampler

    class Colder(SamplingParams):
        @property
        def temperature(self):
            return 0.25

    seen = {}
    monkeypatch.setattr(ops, "sample", lambda logits, tokens, *columns: seen.update(columns=[c.clone() for c in columns]))
    params = [SamplingParams(temperature=0.5 + r, top_k=3 * r or None, top_p=0.9, min_p=0.125, seed=7 + r) for r in range(3)]
    indices = [5, 6, 2**40]
    want = [[0.5, 1.5, 2.5], [0, 3, 6], [0.9] * 3, [0.125] * 3, [7, 8, 9], indices]
    given, places = params, indices
    if collection == "views":
        given, places = dict(enumerate(params)).values(), dict(enumerate(indices)).values()
    elif collection == "others":
        given = [_Others(p) for p in params]
    elif collection == "derived":
        given = params[:2] + [Colder(temperature=2.5, top_k=6, top_p=0.9, min_p=0.125, seed=9)]
        want[0] = [0.5, 1.5, 0.25]
    Sampler("cpu", 4).sample(torch.zeros(3, 8), given, places)
    for column, values in zip(seen["columns"], want):
        assert column[:3].tolist() == torch.tensor(values, dtype=column.dtype).tolist()
