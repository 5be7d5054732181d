"""The tcgen05 attention kernel for wide heads packed side by side, against the ``mma.sync`` kernel
(which takes the same arguments) and the formula in double; and the products per head on the tensor
cores against the CUDA-core kernel."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def formula(q, k, v, position, scale, window, keep, chunk, softcap, sinks, slopes, first_head):
    """One token's rows ``q [G, D]`` against keys and values ``[T, D]`` at positions 0..T-1."""
    place = torch.arange(k.shape[0], device=q.device)
    seen = place <= position
    if window:
        seen &= (position - place < window) | (place < keep)
    if chunk:
        seen &= place >= position - position % chunk
    scores = (q @ k.T) * scale
    if softcap:
        scores = softcap * torch.tanh(scores / softcap)
    heads = torch.arange(first_head, first_head + q.shape[0], device=q.device)
    if slopes is not None:
        scores = scores - slopes[heads].double()[:, None] * (position - place)[None]
    scores = scores.masked_fill(~seen, -math.inf)
    top = scores.max(1, keepdim=True)[0]
    weights = torch.exp(scores - top)
    total = weights.sum(1, keepdim=True)
    if sinks is not None:
        total = total + torch.exp(sinks[heads].double()[:, None] - top)
    return (weights / total) @ v


@pytest.mark.parametrize("head_dim,heads,kv_heads,page,lengths,contexts,options", [
    (256, 32, 1, 16, (70, 1, 9), (0, 200, 131), {}),
    (256, 8, 2, 32, (130,), (3,), dict(window=50, keep_first=5)),
    (192, 3, 1, 64, (1, 1, 1), (0, 63, 64), dict(sinks=True)),       # rows that do not fill a tile
    (160, 64, 1, 16, (5,), (77,), dict(softcap=20.0)),               # two tokens a tile
    (224, 4, 2, 16, (129, 3), (0, 65), dict(slopes=True)),
    (256, 6, 2, 16, (40, 2), (90, 63), dict(chunk=64)),
])
def test_wide_heads_against_the_formula(head_dim, heads, kv_heads, page, lengths, contexts, options):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(head_dim + heads)
    group, options = heads // kv_heads, dict(options)
    total = [c + n for c, n in zip(contexts, lengths)]
    pages = [-(-t // page) for t in total]
    num_pages = sum(pages) + 2
    order = torch.randperm(num_pages)[:sum(pages)].tolist()
    tables = torch.full((len(lengths), max(pages)), -1, dtype=torch.int32)
    k_cache = torch.full((num_pages, kv_heads, head_dim // 8, page, 8), float("nan"))
    v_cache = torch.full_like(k_cache, float("nan"))
    keys, values, at = [], [], 0
    for r, count in enumerate(pages):
        tables[r, :count] = torch.tensor(order[at:at + count], dtype=torch.int32)
        at += count
        k, v = (torch.randn(total[r], kv_heads, head_dim).bfloat16().float() for _ in range(2))
        keys.append(k), values.append(v)
        for t in range(total[r]):
            where = (tables[r, t // page], slice(None), slice(None), t % page)
            k_cache[where] = k[t].view(kv_heads, head_dim // 8, 8)
            v_cache[where] = v[t].view(kv_heads, head_dim // 8, 8)
    n = sum(lengths)
    q = (torch.randn(n, heads * head_dim) * 1.5).bfloat16().cuda()
    starts = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    extra = dict(window=options.get("window", 0), keep_first=options.get("keep_first", 0),
                 chunk=options.get("chunk", 0), softcap=options.get("softcap", 0.0))
    if options.get("sinks"):
        extra["sinks"] = torch.randn(heads).cuda()
    if options.get("slopes"):
        extra["slopes"] = (torch.rand(heads) * 0.1).cuda()
    scale = head_dim ** -0.5
    ints = lambda x: torch.tensor(np.asarray(x, dtype=np.int32)).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for tensor_memory in (None, False):
        out = torch.full((n, heads * head_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.prefill_attention(q, k_cache.bfloat16().cuda(), v_cache.bfloat16().cuda(), ints(starts),
                              ints(contexts), ints(range(len(lengths))), tables.cuda(), out,
                              len(lengths), n, heads, kv_heads, head_dim, page, num_pages, scale, 1,
                              status, query_lengths=list(lengths), packed=True,
                              tensor_memory=tensor_memory, **extra)
        outs.append(out.double())
    assert int(status.item()) == 0
    want = torch.empty(n, heads, head_dim, dtype=torch.float64, device="cuda")
    for r, length in enumerate(lengths):
        for t in range(length):
            for kv in range(kv_heads):
                rows = slice(kv * group, (kv + 1) * group)
                want[starts[r] + t, rows] = formula(
                    q[starts[r] + t].double().view(heads, head_dim)[rows],
                    keys[r][:, kv].double().cuda(), values[r][:, kv].double().cuda(),
                    contexts[r] + t, scale, extra["window"], extra["keep_first"], extra["chunk"],
                    extra["softcap"], extra.get("sinks"), extra.get("slopes"), kv * group)
    want = want.view(n, -1)
    for out in outs:
        assert torch.isfinite(out).all()
        # the result is stored in bfloat16 (2^-9 of it), the probabilities carry 16 bits
        assert ((out - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all()


@pytest.mark.parametrize("tokens,heads,in_dim,out_dim,x_stride,out_stride", [
    (33, 3, 64, 40, 72, 40), (129, 2, 192, 128, 256, 128), (300, 5, 128, 300, 128, 304),
    (1100, 40, 64, 256, 64, 256),      # more tiles than SMs
    (257, 1, 64, 500, 72, 512),        # one head: pairs of CTAs, tiles in pieces
    (1, 32, 128, 192, 128, 256), (1, 1, 64, 8, 64, 8), (5, 3, 192, 128, 256, 128), (16, 40, 64, 40, 72, 48),
    (17, 2, 128, 300, 136, 304), (32, 32, 192, 128, 256, 128),
])
def test_products_per_head_on_the_tensor_cores(tokens, heads, in_dim, out_dim, x_stride, out_stride):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens)
    x = torch.randn(tokens + 3, heads * x_stride).bfloat16().cuda()
    x[tokens:] = float("nan")
    w = torch.randn(heads, out_dim, in_dim).bfloat16().cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((tokens + 3, heads * out_stride + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    plain = out.clone()
    ops.head_products(x, x_stride, w, out, out_stride, tokens, status)
    ops.head_products(x, x_stride, w, plain, out_stride, tokens)
    assert int(status.item()) == 0
    want = torch.einsum("thi,hoi->tho", x[:tokens].double().view(tokens, heads, x_stride)[..., :in_dim],
                        w.double())
    for got in (out, plain):
        assert (got[tokens:] == 7.0).all()
        part = got[:tokens, :heads * out_stride].view(tokens, heads, out_stride)
        assert (part[..., out_dim:] == 7.0).all()
        error = (part[..., :out_dim].double() - want).abs()
        # one rounding to bfloat16 of a float32 sum of in_dim products
        assert (error <= 2.0 ** -8 * want.abs() + in_dim * 2.0 ** -20).all()


def test_the_same_heads_are_packed_as_before():
    from helix_runtime_b200.ops import library as ops
    tokens = ops.lib().hx_prefill_attention_tc_packed_tokens
    for heads, kv_heads in ((32, 1), (64, 1), (65, 1), (4, 4), (6, 2), (7, 2)):
        before = ops.prefill_attention_packed_tokens(heads, kv_heads)
        assert tokens(heads, kv_heads, 256, 16) == (128 // (heads // kv_heads) if before else 0)
    assert tokens(32, 1, 128, 16) == tokens(32, 1, 240, 16) == tokens(32, 1, 256, 8) == 0


@pytest.mark.parametrize("head_dim,value_dim", [(160, 32), (160, 96), (192, 160), (256, 192), (256, 224)])
@pytest.mark.parametrize("page_size", [16, 32])
def test_leading_columns_of_the_values(head_dim, value_dim, page_size):
    """So many columns as are asked for are those of the whole call, bit for bit; the others stay.  (Contexts
    of one tile, of an odd and an even number of tiles, and a window that begins inside one.)"""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(head_dim + value_dim)
    heads, lengths, contexts = 8, (70, 3, 20), (0, 130, 61)
    pages_of = [-(-(length + context) // page_size) for length, context in zip(lengths, contexts)]
    pages = sum(pages_of)
    q = torch.randn(sum(lengths), heads * head_dim, device="cuda").bfloat16()
    keys = torch.randn(pages, 1, page_size * head_dim, device="cuda").bfloat16()
    values = torch.randn_like(keys)
    table = torch.zeros(len(lengths), max(pages_of), dtype=torch.int32)
    order, at = torch.randperm(pages).int(), 0
    for request, count in enumerate(pages_of):
        table[request, :count] = order[at:at + count]
        at += count
    starts = torch.tensor([0, *torch.tensor(lengths).cumsum(0)], dtype=torch.int32).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for window in (0, 50):
        outs = []
        for wanted in (0, value_dim):
            out = torch.full((sum(lengths), heads * head_dim), 5.0, device="cuda").bfloat16()
            ops.prefill_attention(q, keys, values, starts, torch.tensor(contexts, dtype=torch.int32).cuda(),
                                  torch.arange(len(lengths), dtype=torch.int32).cuda(), table.cuda(), out,
                                  len(lengths), sum(lengths), heads, 1, head_dim, page_size, pages,
                                  head_dim ** -0.5, 1, status, query_lengths=lengths, window=window,
                                  packed=True, value_dim=wanted)
            outs.append(out.view(-1, heads, head_dim))
        whole, part = outs
        assert torch.equal(part[..., :value_dim], whole[..., :value_dim])
        assert (part[..., value_dim:] == 5.0).all() and whole.float().abs().max() < 5.0
    assert int(status.item()) == 0
