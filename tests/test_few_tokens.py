"""A layer's products for a few tokens against the separate kernels' plain statements, at the edges of what the
kernels take: 1, 8, 9 and 16 tokens, K of one piece a warp and of a remainder, rows of one group, a page table with
padding and a bad page."""
import pytest
import torch

import kernel_references as ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda:0")


def _normed(h, weight, eps):
    return h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + eps) * weight


def _close(got, want, k):
    # one operand rounded to bfloat16 (2^-9 of a term, independently) under sums of k terms, the result once more: both in
    # proportion to the root mean square of what was stored (the places of a cache that nothing was written to aside)
    written = want != 0
    bound = 2 ** -8 * want[written].double().pow(2).mean().sqrt().item()
    # (a product of two branches has values of twenty times that: rounding one to bfloat16 is 2^-9 of it, and either
    # branch's own error enters times the other)
    error = ((got.double() - want.double()).abs() - 2 ** -8 * want.double().abs()).clamp_min(0)[written]
    assert float(error.max()) < 6 * bound and float(error.pow(2).mean().sqrt()) < bound, (k, float(error.max()), bound)


@pytest.mark.parametrize("tokens,hidden,heads,kv_heads,size,rotary,pending", [
    (1, 896, 14, 2, 64, True, True), (8, 896, 14, 2, 64, True, True), (9, 896, 14, 2, 64, True, False),
    (16, 1024, 12, 2, 128, True, True), (3, 32, 2, 1, 16, True, True), (5, 288, 3, 3, 48, False, True), (16, 992, 4, 4, 32, True, False),
])
def test_norm_qkv_rotation_and_store(dev, tokens, hidden, heads, kv_heads, size, rotary, pending):
    from einf_b200 import ops

    torch.manual_seed(tokens + hidden)
    rows, page = (heads + 2 * kv_heads) * size, 16
    residual = torch.randn(tokens, hidden, device=dev) * 3
    extra = torch.randn(tokens, hidden, device=dev) if pending else None
    norm = torch.randn(hidden, device=dev) * 0.1 + 1
    weight = (torch.randn(rows, hidden, device=dev) * hidden ** -0.5).bfloat16()
    bias = torch.randn(rows, device=dev) if pending else None
    positions = torch.randint(0, 30000, (tokens,), dtype=torch.int32, device=dev)
    inv_freq = 1.0 / (1e6 ** (torch.arange(0, size, 2, device=dev).float() / size)) if rotary else torch.empty(0, device=dev)
    slots = torch.randperm(4 * page, device=dev)[:tokens].to(torch.int32)
    if tokens > 2:
        slots[1] = -1
    caches = [torch.zeros(4, kv_heads, page, size, dtype=torch.bfloat16, device=dev) for _ in range(4)]
    q, want_q = (torch.zeros(tokens, heads, size, dtype=torch.bfloat16, device=dev) for _ in range(2))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    before = residual.clone()
    ops.few_qkv(residual, extra, norm, 1e-6, weight, bias, positions, inv_freq, slots, q, caches[0], caches[1], heads, kv_heads,
                size, status)
    assert torch.equal(residual, before) and int(status) == 0
    h = residual + extra if pending else residual
    qkv = (_normed(h.double(), norm.double(), 1e-6) @ weight.double().T).float()
    ref.rope_kv_write(qkv, bias, positions, inv_freq, slots, want_q, caches[2], caches[3], heads, kv_heads, size, status)
    _close(q, want_q, hidden)
    _close(caches[0], caches[2], hidden)
    _close(caches[1], caches[3], hidden)
    assert torch.equal(caches[0] == 0, caches[2] == 0)
    slots[0] = 4 * page + 3          # a page beyond the pool is reported, nothing is written for it
    ops.few_qkv(residual, extra, norm, 1e-6, weight, bias, positions, inv_freq, slots, q, caches[0], caches[1], heads, kv_heads,
                size, status)
    assert int(status) == ops.STATUS_BAD_PAGE
    ops.few_qkv(residual, extra, norm, 1e-6, weight, bias, positions, inv_freq, None, q, None, None, heads, kv_heads, size, status)
    _close(q, want_q, hidden)


@pytest.mark.parametrize("tokens,hidden,inter", [(1, 896, 4864), (8, 896, 4864), (9, 64, 16), (16, 1024, 4096), (2, 992, 48)])
def test_norm_gate_up_and_silu(dev, tokens, hidden, inter):
    from einf_b200 import ops

    torch.manual_seed(tokens + inter)
    residual = torch.randn(tokens, hidden, device=dev) * 2
    norm = torch.randn(hidden, device=dev) * 0.1 + 1
    weight = (torch.randn(2 * inter, hidden, device=dev) * hidden ** -0.5).bfloat16()
    out, status = torch.empty(tokens, inter, dtype=torch.bfloat16, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    ops.few_gate_up(residual, norm, 1e-6, weight, out, status)
    both = _normed(residual.double(), norm.double(), 1e-6) @ weight.double().T
    _close(out, torch.nn.functional.silu(both[:, :inter]) * both[:, inter:], hidden)
    assert int(status) == 0


@pytest.mark.parametrize("tokens,k,rows", [(1, 896, 896), (8, 4864, 896), (9, 4864, 896), (16, 32, 8), (16, 2080, 1536), (5, 5120, 1024), (12, 288, 24)])
def test_product_into_the_stream_and_alone(dev, tokens, k, rows):
    from einf_b200 import ops

    torch.manual_seed(k + rows)
    x = torch.randn(tokens, k, device=dev).bfloat16()
    weight = (torch.randn(rows, k, device=dev) * k ** -0.5).bfloat16()
    want = x.double() @ weight.double().T
    out, status = torch.empty(tokens, rows, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    ops.few_product(x, weight, out, status)
    # no rounding but that of 32-bit sums of k terms, cut off by the instruction
    torch.testing.assert_close(out.double(), want, rtol=0, atol=k * 2 ** -24 * 4)
    stream, pending = torch.randn(tokens, rows, device=dev), torch.randn(tokens, rows, device=dev)
    for added in (pending, None):
        got = stream.clone()
        ops.few_product(x, weight, got, status, add_to_stream=True, pending=added)
        assert torch.allclose(got, stream + out + (0 if added is None else added), rtol=0, atol=2e-6)
    assert int(status) == 0


@pytest.mark.parametrize("rotary", [False, True])
def test_a_value_that_is_not_finite_stays_in_its_element(dev, rotary):
    """Values, and heads that are not rotated, do not meet the other half of their head."""
    from einf_b200 import ops

    torch.manual_seed(11)
    tokens, hidden, heads, kv_heads, size, page = 3, 64, 2, 1, 32, 16
    residual, norm = torch.randn(tokens, hidden, device=dev), torch.ones(hidden, device=dev)
    weight = (torch.randn((heads + 2 * kv_heads) * size, hidden, device=dev) * 0.1).bfloat16()
    bias = torch.zeros(weight.shape[0], device=dev)
    inv_freq = 1.0 / (1e4 ** (torch.arange(0, size, 2, device=dev).float() / size)) if rotary else torch.empty(0, device=dev)
    marked = {"q": 5, "k": heads * size + 20, "v": (heads + kv_heads) * size + 3}
    for value in (float("inf"), float("nan")):
        for place in marked.values():
            bias[place] = value
        q = torch.zeros(tokens, heads, size, dtype=torch.bfloat16, device=dev)
        k, v = (torch.zeros(1, kv_heads, page, size, dtype=torch.bfloat16, device=dev) for _ in range(2))
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        ops.few_qkv(residual, None, norm, 1e-6, weight, bias, torch.arange(1, tokens + 1, dtype=torch.int32, device=dev), inv_freq,
                    torch.arange(tokens, dtype=torch.int32, device=dev), q, k, v, heads, kv_heads, size, status)
        rows = {"q": q.view(tokens, -1), "k": k[0, 0, :tokens], "v": v[0, 0, :tokens]}
        for name, first in (("q", 0), ("k", heads * size), ("v", (heads + kv_heads) * size)):
            at = marked[name] - first
            bad = {at, at + size // 2 if at % size < size // 2 else at - size // 2} if rotary and name != "v" else {at}
            assert set((~torch.isfinite(rows[name])).any(0).nonzero().flatten().tolist()) == bad, (name, value)


def test_a_token_gets_the_same_in_every_batch(dev):
    """A token's sums do not depend on the tokens beside it."""
    from einf_b200 import ops

    torch.manual_seed(3)
    residual, norm = torch.randn(16, 896, device=dev), torch.ones(896, device=dev)
    weight = (torch.randn(9728, 896, device=dev) * 0.03).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    results = []
    for tokens in (1, 8, 9, 16):
        out = torch.empty(tokens, 4864, dtype=torch.bfloat16, device=dev)
        ops.few_gate_up(residual[:tokens].contiguous(), norm, 1e-6, weight, out, status)
        results.append(out[0])
    assert all(torch.equal(results[0], r) for r in results[1:])


def test_sizes_that_are_refused(dev):
    from einf_b200 import ops

    status = torch.zeros(1, dtype=torch.int32, device=dev)
    x, weight = torch.zeros(17, 64, dtype=torch.bfloat16, device=dev), torch.zeros(8, 64, dtype=torch.bfloat16, device=dev)
    with pytest.raises(ops.UnsupportedSize):
        ops.few_product(x, weight, torch.zeros(17, 8, device=dev), status)
    with pytest.raises(ops.UnsupportedSize):
        ops.few_product(x[:2, :40].contiguous(), weight[:, :40].contiguous(), torch.zeros(2, 8, device=dev), status)
