"""Attention of a prompt chunk on tcgen05 (flash_umma.cuh) against plain 64-bit attention on the same rows."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def plain(q, keys, values, scale, visible, bias=None, sink=None):
    """q [T, H, d]; keys [S, G, d] and values [S, G, dv] by position; visible [T, S]; bias [H, T, S]; sink [H]."""
    share = q.shape[1] // keys.shape[1]
    k, v = keys.double().repeat_interleave(share, 1), values.double().repeat_interleave(share, 1)
    s = torch.einsum("thd,shd->hts", q.double(), k) * scale
    if bias is not None:
        s = s + bias
    s = s.masked_fill(~visible, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(-1, s.shape[1], 1)], -1)
    p = torch.softmax(s, -1)[..., :keys.shape[0]]
    return torch.einsum("hts,shd->thd", p, v)


def close(got, want, rounds):
    """Per row: exact products and fp32 sums; ``rounds`` bf16 roundings (2^-8 each) of probabilities, result and factors."""
    worst = (got.double() - want).abs().amax(-1) / want.abs().amax(-1)
    assert float(worst.max()) < rounds * 2.0 ** -8, float(worst.max())


@pytest.mark.parametrize("tokens,position,heads,kv_heads", [
    (40, 0, 16, 2), (41, 0, 16, 2), (20, 20, 8, 8), (21, 20, 8, 8), (2, 39, 16, 2),               # both sides of the line between the forms
    (2, 0, 16, 2), (16, 0, 16, 2), (17, 63, 16, 2), (65, 0, 16, 2), (200, 1000, 16, 2), (130, 3, 6, 2), (300, 0, 2, 2), (129, 64, 4, 1), (2048, 37, 16, 2)])
def test_gated_attention_of_a_chunk(cuda_device, tokens, position, heads, kv_heads):
    from quickdraw_b200._lib import call, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    new = lambda *shape, std=1.0: (torch.randn(shape, generator=gen, device=cuda_device) * std).to(BF16)
    capacity = position + tokens + 3
    keys, values = new(capacity, kv_heads, 256, std=2.0), new(capacity, kv_heads, 256)
    keys[position + tokens:], values[position + tokens:] = float("nan"), float("nan")          # not written yet
    qg, k, v = new(tokens, heads * 512), new(tokens, kv_heads * 256), new(tokens, kv_heads * 256)
    norm = torch.zeros(256, dtype=BF16, device=cuda_device)
    q, out = torch.empty(tokens, heads, 256, dtype=BF16, device=cuda_device), torch.empty(tokens, heads, 256, dtype=BF16, device=cuda_device)
    call("qd_seq_attention", ptr(qg), ptr(k), ptr(v), ptr(norm), ptr(norm), ptr(keys), ptr(values), ptr(q), ptr(out), tokens, position, capacity,
         heads, kv_heads, 256, 64, 1e6, 1e-6, stream_of(q))
    end = position + tokens
    at = torch.arange(position, end, device=cuda_device)
    visible = torch.arange(end, device=cuda_device)[None] <= at[:, None]
    want = plain(q, keys[:end], values[:end], 0.0625, visible) * torch.sigmoid(qg.view(tokens, heads, 2, 256)[:, :, 1].double())
    close(out, want, 4)


@pytest.mark.parametrize("tokens,position,heads,kv_heads,shared,span,capacity,chunked,slopes,sink,gate", [
    (300, 0, 16, 4, 0, 1024, 300, False, False, 1, 1),          # windowed, learned sinks, a gate per head
    (700, 100, 8, 2, 0, 100, 900, False, False, 1, 1),          # ... a short window: leading tiles that later rows do not see
    (513, 2000, 8, 8, 64, 256, 1024, False, False, 0, 2),       # shared key columns, a gate per column, the ring wraps
    (400, 700, 16, 4, 0, 256, 1024, True, True, 2, 0),          # chunks, distance penalty, a zero sink
    (129, 0, 3, 1, 0, 64, 256, True, True, 2, 0),               # heads that do not divide a row tile
    (1200, 5, 4, 4, 64, 5000, 1300, False, False, 0, 2),
])
def test_bounded_attention_of_a_chunk(cuda_device, tokens, position, heads, kv_heads, shared, span, capacity, chunked, slopes, sink, gate):
    from ctypes import byref

    from quickdraw_b200._lib import AttentionArgs, call_hybrid, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    new = lambda *shape, std=1.0: (torch.randn(shape, generator=gen, device=cuda_device) * std).to(BF16)
    first, end = max(0, position - span + 1), position + tokens
    keys, values, common = new(end, kv_heads, 128, std=2.0), new(end, kv_heads, 128), new(end, shared)
    ring = lambda t: torch.full((capacity, *t.shape[1:]), float("nan"), dtype=BF16, device=cuda_device)
    kr, vr, cr = ring(keys), ring(values), ring(common)
    for j in range(max(first, end - capacity), end):
        kr[j % capacity], vr[j % capacity], cr[j % capacity] = keys[j], values[j], common[j]
    q, gates = new(tokens, heads, 128 + shared), new(tokens, heads * (128 if gate == 2 else 1))
    slope = torch.rand(heads, generator=gen, device=cuda_device) * 0.05
    sinks, out = new(heads), torch.empty(tokens, heads, 128, dtype=BF16, device=cuda_device)
    scale = (128 + shared) ** -0.5
    args = AttentionArgs(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, shared_dim=shared, scale=scale, ld_k=kv_heads * 128, ld_v=kv_heads * 128,
                         ld_shared=shared, k_cache=ptr(kr), v_cache=ptr(vr), k_shared=ptr(cr) if shared else None, q_rows=ptr(q), out=ptr(out),
                         gate=ptr(gates), ld_gate=gates.shape[1], gate_kind=gate, sink=ptr(sinks), sink_kind=sink,
                         slopes=ptr(slope) if slopes else None, mask=int(chunked), span=min(span, capacity), capacity=capacity, position=position,
                         tokens=tokens, dtype=0)
    call_hybrid("qd_attention", byref(args), stream_of(q))
    at, j = torch.arange(position, end, device=cuda_device)[:, None], torch.arange(end, device=cuda_device)[None]
    visible = (j <= at) & (j >= (at - at % span if chunked else at - span + 1))
    bias = -slope.double()[:, None, None] * (at - j) if slopes else None
    with_shared = torch.cat([keys, common[:, None].expand(-1, kv_heads, -1)], -1)
    extra = {0: None, 1: sinks, 2: torch.zeros(heads, device=cuda_device)}[sink]
    want = plain(q, with_shared, values, scale, visible, bias, extra)
    if gate:
        want = want * torch.sigmoid(gates.double().view(tokens, heads, -1))
    close(out, want, 1.5)


@pytest.mark.parametrize("tokens,position", [(64, 0), (511, 0), (200, 3000)])
def test_chunk_attention_rounds_its_result_only(cuda_device, tokens, position):
    """Sharp scores, gates of one: with probabilities of sixteen bits the distance to 64 bits is that of one bf16 rounding
    of the result (their own part is 2^-18 of it, below a hundredth); eight bits add a quarter."""
    from quickdraw_b200._lib import call, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).to(BF16)
    end = position + tokens
    keys, values, qg = new(end, 2, 256), new(end, 2, 256), new(tokens, 16, 2, 256)
    qg[:, :, 1] = 30.0
    k, v, norm, q_norm = new(tokens, 512), new(tokens, 512), torch.zeros(256, dtype=BF16, device=cuda_device), torch.full((256,), 3.0, dtype=BF16, device=cuda_device)
    q, out = torch.empty(tokens, 16, 256, dtype=BF16, device=cuda_device), torch.empty(tokens, 16, 256, dtype=BF16, device=cuda_device)
    call("qd_seq_attention", ptr(qg), ptr(k), ptr(v), ptr(q_norm), ptr(norm), ptr(keys), ptr(values), ptr(q), ptr(out), tokens, position, end,
         16, 2, 256, 64, 1e6, 1e-6, stream_of(q))
    at = torch.arange(position, end, device=cuda_device)
    want = plain(q, keys, values, 0.0625, torch.arange(end, device=cuda_device)[None] <= at[:, None])
    error = lambda t: float((t.double() - want).norm() / want.norm())
    assert error(out) < 1.01 * error(want.to(BF16)), (error(out), error(want.to(BF16)))


@pytest.mark.parametrize("tokens,position,heads,kv_heads,span,capacity", [
    (200, 30, 16, 2, 0, 240),           # the gated form, head dimension 256
    (300, 100, 8, 2, 64, 512),          # a window: masked keys on both sides, whole tiles and partial ones
    (150, 900, 4, 4, 100, 256),         # ... whose ring wraps
])
def test_values_that_are_not_finite_reach_those_who_see_them(cuda_device, tokens, position, heads, kv_heads, span, capacity):
    """An infinity and a NaN among a chunk's values: rows that do not see their tokens are what they were, the others are infinite or
    NaN in that column alone."""
    from ctypes import byref

    from quickdraw_b200._lib import AttentionArgs, call, call_hybrid, ptr, stream_of
    dim, end = 128 if span else 256, position + tokens
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).to(BF16)
    keys, values, q, qg = new(end, kv_heads, dim), new(end, kv_heads, dim), new(tokens, heads, dim), new(tokens, heads, 2, dim)

    def attend(values):
        out = torch.empty(tokens, heads, dim, dtype=BF16, device=cuda_device)
        kr, vr = (torch.zeros(capacity, kv_heads, dim, dtype=BF16, device=cuda_device) for _ in range(2))
        for j in range(max(0, end - capacity), end):
            kr[j % capacity], vr[j % capacity] = keys[j], values[j]
        if span:
            args = AttentionArgs(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, shared_dim=0, scale=dim ** -0.5, ld_k=kv_heads * dim,
                                 ld_v=kv_heads * dim, k_cache=ptr(kr), v_cache=ptr(vr), q_rows=ptr(q), out=ptr(out), gate=ptr(q), ld_gate=8, gate_kind=0,
                                 sink_kind=0, mask=0, span=span, capacity=capacity, position=position, tokens=tokens, dtype=0)
            call_hybrid("qd_attention", byref(args), stream_of(q))
        else:
            norm, rows = torch.zeros(dim, dtype=BF16, device=cuda_device), torch.empty_like(q)
            fresh = [t[position:].reshape(tokens, -1).contiguous() for t in (keys, values)]
            call("qd_seq_attention", ptr(qg), *map(ptr, fresh), ptr(norm), ptr(norm), ptr(kr), ptr(vr), ptr(rows), ptr(out), tokens, position,
                 capacity, heads, kv_heads, dim, 64, 1e6, 1e-6, stream_of(q))
        return out

    plainly, share = attend(values), heads // kv_heads
    bad = [(position + 20, 0, 5, float("inf")), (position + tokens - 10, kv_heads - 1, dim - 1, float("nan")), (position + 83, 0, 70, float("-inf"))]
    want = plainly.clone()
    for j, g, column, value in bad:
        values[j, g, column] = value
        last = min(tokens, j - position + span) if span else tokens
        want[j - position:last, g * share:(g + 1) * share, column] = value
    got = attend(values)
    finite = want.isfinite()
    # (Sums done again in fp32 may round to the other neighbour, which is a bf16 spacing, at most 2^-7; the gated form rounds twice, the
    # attended value and its product with the gate: two spacings.  And 2^-17 of the sum of magnitudes.)
    torch.testing.assert_close(got[finite], want[finite], rtol=2 ** -7 if span else 2 ** -6, atol=2 ** -17 * float(values[values.isfinite()].abs().max()))
    assert torch.equal(got.isnan(), want.isnan())
    assert bool((got[~finite & ~want.isnan()] == want[~finite & ~want.isnan()]).all())


@pytest.mark.parametrize("dim,shared,heads,kv_heads,wider,tokens,position,span,capacity", [
    (96, 32, 8, 2, 0, 90, 10, 50, 256),           # shared columns inside a box of 64: rows copied one by one
    (136, 56, 4, 4, 8, 70, 0, 300, 300),          # ... and rows wider than their heads
    (64, 128, 6, 2, 64, 200, 100, 70, 320),       # shared columns in boxes of their own
    (128, 0, 8, 2, 24, 300, 500, 128, 512),       # wider rows through boxes
    (128, 64, 4, 1, 0, 20, 33, 20, 40),           # a ring below a tile
    (192, 0, 2, 2, 0, 33, 7, 64, 100),
])
def test_forms_of_rows_that_a_chunk_may_have(cuda_device, dim, shared, heads, kv_heads, wider, tokens, position, span, capacity):
    """Every split of the key columns between a head's own and shared ones, strides, rings: what the dispatch takes to tcgen05."""
    from ctypes import byref

    from quickdraw_b200._lib import AttentionArgs, call_hybrid, ptr, stream_of
    gen = torch.Generator(device=cuda_device).manual_seed(dim)
    new = lambda *shape: torch.randn(shape, generator=gen, device=cuda_device).to(BF16)
    end = position + tokens
    keys, values, common, q = new(end, kv_heads, dim), new(end, kv_heads, 128), new(end, shared), new(tokens, heads, dim + shared)
    rings = []
    for rows in (keys, values, common):
        flat = rows.reshape(end, -1)
        ring = torch.full((capacity, flat.shape[1] + wider), float("nan"), dtype=BF16, device=cuda_device)
        for j in range(max(0, end - capacity), end):
            ring[j % capacity, :flat.shape[1]] = flat[j]
        rings.append(ring)
    out = torch.empty(tokens, heads, 128, dtype=BF16, device=cuda_device)
    scale = (dim + shared) ** -0.5
    args = AttentionArgs(heads=heads, kv_heads=kv_heads, dim=dim, vdim=128, shared_dim=shared, scale=scale, ld_k=rings[0].shape[1], ld_v=rings[1].shape[1],
                         ld_shared=rings[2].shape[1], k_cache=ptr(rings[0]), v_cache=ptr(rings[1]), k_shared=ptr(rings[2]) if shared else None,
                         q_rows=ptr(q), out=ptr(out), gate=None, ld_gate=8, gate_kind=0, sink_kind=0, mask=0, span=span, capacity=capacity,
                         position=position, tokens=tokens, dtype=0)
    call_hybrid("qd_attention", byref(args), stream_of(q))
    at, j = torch.arange(position, end, device=cuda_device)[:, None], torch.arange(end, device=cuda_device)[None]
    close(out, plain(q, torch.cat([keys, common[:, None].expand(-1, kv_heads, -1)], -1), values, scale, (j <= at) & (j > at - span)), 1.5)


@pytest.mark.parametrize("tokens,position,heads,kv_heads,shared,span,capacity,chunked,slopes,sink,gate,bad", [
    (300, 0, 16, 4, 0, 1024, 300, False, False, 1, 1, None), (700, 100, 8, 2, 0, 100, 900, False, False, 1, 1, None),
    (593, 2000, 8, 8, 64, 256, 1024, False, False, 0, 2, None), (400, 700, 16, 4, 0, 256, 1024, True, True, 2, 0, None),
    (1601, 0, 3, 1, 0, 33, 1700, True, True, 2, 0, None), (1200, 5, 4, 4, 64, 5000, 1300, False, False, 0, 2, None),
    (600, 50, 8, 2, 64, 64, 700, False, False, 0, 0, math.inf), (500, 0, 12, 4, 0, 5000, 500, False, False, 1, 2, math.nan)])
def test_bounded_attention_of_an_fp32_chunk(cuda_device, tokens, position, heads, kv_heads, shared, span, capacity, chunked, slopes, sink, gate, bad):
    """Operands as three bf16 pieces: masks, rings that wrap, rows for the one and the other group of warps alone, everything that may stand
    around the softmax, values that are not finite.  fp32 sums of some 128 and 1000 terms and scores of about ten: 2e-6."""
    from ctypes import byref

    from quickdraw_b200._lib import AttentionArgs, call_hybrid, ptr, stream_of
    assert tokens * heads >= 32 * 148
    gen = torch.Generator(device=cuda_device).manual_seed(tokens)
    new = lambda *shape, std=1.0: torch.randn(shape, generator=gen, device=cuda_device) * std
    first, end = max(0, position - span + 1), position + tokens
    keys, values, common = new(end, kv_heads, 128, std=2.0), new(end, kv_heads, 128), new(end, shared)
    spoilt = values.clone()
    if bad is not None:
        spoilt[position + 201, 0, 7] = bad
    ring = lambda t: torch.full((capacity, *t.shape[1:]), float("nan"), device=cuda_device)
    kr, vr, cr = ring(keys), ring(values), ring(common)
    for j in range(max(first, end - capacity), end):
        kr[j % capacity], vr[j % capacity], cr[j % capacity] = keys[j], spoilt[j], common[j]
    q, gates = new(tokens, heads, 128 + shared), new(tokens, heads * (128 if gate == 2 else 1))
    slope = torch.rand(heads, generator=gen, device=cuda_device) * 0.05
    sinks, out = new(heads).to(BF16), torch.full((tokens, heads, 128), float("nan"), device=cuda_device)
    scale = (128 + shared) ** -0.5
    args = AttentionArgs(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, shared_dim=shared, scale=scale, ld_k=kv_heads * 128, ld_v=kv_heads * 128,
                         ld_shared=shared, k_cache=ptr(kr), v_cache=ptr(vr), k_shared=ptr(cr) if shared else None, q_rows=ptr(q), out=ptr(out),
                         gate=ptr(gates), ld_gate=gates.shape[1], gate_kind=gate, sink=ptr(sinks), sink_kind=sink,
                         slopes=ptr(slope) if slopes else None, mask=int(chunked), span=min(span, capacity), capacity=capacity, position=position,
                         tokens=tokens, dtype=1)
    call_hybrid("qd_attention", byref(args), stream_of(q))
    at, j = torch.arange(position, end, device=cuda_device)[:, None], torch.arange(end, device=cuda_device)[None]
    visible = (j <= at) & (j >= (at - at % span if chunked else at - span + 1))
    bias = -slope.double()[:, None, None] * (at - j) if slopes else None
    with_shared = torch.cat([keys, common[:, None].expand(-1, kv_heads, -1)], -1)
    extra = {0: None, 1: sinks, 2: torch.zeros(heads, device=cuda_device)}[sink]
    want = plain(q, with_shared, values, scale, visible, bias, extra)
    if gate:
        want = want * torch.sigmoid(gates.double().view(tokens, heads, -1))
    kept = torch.ones_like(want, dtype=torch.bool)
    if bad is not None:
        kept[:, :heads // kv_heads, 7] = ~visible[:, position + 201, None]
        assert not torch.isfinite(out[~kept]).any()
    assert float((out.double() - want)[kept].norm() / want[kept].norm()) < 2e-6


@pytest.mark.parametrize("heads,kv_heads,shared", [(16, 4, 0), (16, 16, 64)])
def test_bounded_attention_of_an_fp32_chunk_at_the_end_of_the_range(cuda_device, heads, kv_heads, shared):
    """Keys and queries with infinities and with the largest number, products that pass it, values of the largest number: what plain fp32 sums
    give.  A key whose score is minus infinity has weight zero and touches nothing, one of plus infinity or NaN spoils the rows that see it, a
    masked one none.  fp32 sums as in the test above: 2e-6; a row that weighs one huge value: as an fp32 product."""
    from ctypes import byref

    from quickdraw_b200._lib import AttentionArgs, call_hybrid, ptr, stream_of
    tokens, span, largest = 320, 150, torch.finfo(torch.float32).max
    gen = torch.Generator(device=cuda_device).manual_seed(heads)
    new = lambda *shape, std=1.0: torch.randn(shape, generator=gen, device=cuda_device) * std
    keys, values, common, q = new(tokens, kv_heads, 128, std=2.0), new(tokens, kv_heads, 128), new(tokens, shared), new(tokens, heads, 128 + shared)
    q[..., 0] = q[..., 0].abs() + 0.1
    q[..., 1] = 0.0
    keys[..., 0], keys[..., 1] = keys[..., 0] * 0.01, 0.0
    keys[20, 0, 0] = -math.inf                     # weight zero for all that see it
    keys[40, 0, 0] = -largest                      # a product of it and 4 passes the largest number: weight zero too
    q[40:190, :heads // kv_heads, 0] += 4.0
    keys[60, 1, 0] = math.inf                      # plus infinity: rows 60 .. 209 of key/value head 1
    q[250, 2 * heads // kv_heads, 1] = math.inf    # a query: infinity times zero is NaN
    keys[301, 3, 1] = -largest                     # times zero: nothing
    values[5, 0, 9], values[310, 2, 3] = -largest, largest
    args = dict(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, shared_dim=shared, scale=(128 + shared) ** -0.5, ld_k=kv_heads * 128, ld_v=kv_heads * 128,
                ld_shared=shared, k_cache=ptr(keys), v_cache=ptr(values), k_shared=ptr(common) if shared else None, gate=None, ld_gate=8, gate_kind=0,
                sink_kind=0, mask=0, span=span, capacity=tokens, position=0, tokens=tokens, dtype=1)
    out = torch.full((tokens, heads, 128), float("nan"), device=cuda_device)
    call_hybrid("qd_attention", byref(AttentionArgs(q_rows=ptr(q), out=ptr(out), **args)), stream_of(q))
    at, j = torch.arange(tokens, device=cuda_device)[:, None], torch.arange(tokens, device=cuda_device)[None]
    share = heads // kv_heads
    k = torch.cat([keys, common[:, None].expand(-1, kv_heads, -1)], -1).repeat_interleave(share, 1).double()
    v = values.repeat_interleave(share, 1).double()
    terms = torch.einsum("thd,jhd->htj", q.double(), k)
    terms = torch.where(terms.abs() > largest, terms.sign() * math.inf, terms)
    scores = (terms * (128 + shared) ** -0.5).masked_fill(~((j <= at) & (j > at - span)), -math.inf)
    weights = torch.softmax(scores, -1)
    want = torch.einsum("htj,jhd->thd", weights, v)
    spoilt = weights.isnan().any(-1).T
    assert int(spoilt.sum()) == 150 * share + 1
    assert bool(out[spoilt].isnan().all()) and bool(out[~spoilt].isfinite().all())
    huge = torch.zeros_like(want, dtype=torch.bool)
    huge[5:5 + span, :share, 9] = True
    huge[310:, 2 * share:3 * share, 3] = True
    plain_ones = ~huge & ~spoilt[..., None]
    assert float((out.double() - want)[plain_ones].norm() / want[plain_ones].norm()) < 2e-6
    assert float(((out.double() - want)[huge & ~spoilt[..., None]] / largest).abs().max()) < 1e-6
