"""Small kernels of prompt layers that work in pieces of several numbers, at the edges of their pieces and
runs, against the same sums in double or against the road of single numbers."""
from __future__ import annotations

import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,channels", [
    ((1, 2, 3, 4, 5, 6, 7), 8), ((1,) * 9, 40), ((2,), 2056), ((3, 1, 1, 1, 40, 2, 1), 264),
    ((2049,), 4096), ((700, 2, 1, 500, 3), 2048),
])
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_causal_filter(lengths, channels, taps):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(taps)
    tokens, reach = sum(lengths), taps - 1
    starts = [0, *itertools.accumulate(lengths)]
    raw = torch.randn(tokens, channels + 8, device="cuda").bfloat16()[:, :channels]
    sums = torch.randn(tokens, channels + 4, device="cuda")[:, :channels]
    weight = torch.randn(channels, taps, device="cuda")
    bias, in_bias = torch.randn(2, channels, device="cuda")
    before = torch.randn(len(lengths) + 1, max(1, reach) * channels, device="cuda")
    token_request = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).int().cuda()
    slots = torch.arange(len(lengths), 0, -1, dtype=torch.int32, device="cuda")
    for rows, silu, biased in ((raw, True, False), (raw, False, True), (sums, True, False), (sums, False, True)):
        out = torch.zeros(tokens, channels, device="cuda").bfloat16()
        state = before.clone()
        ops.causal_filter(rows, out, weight, bias, state if taps > 1 else None, tokens, silu, token_request,
                          slots, torch.tensor(starts, dtype=torch.int32).cuda(),
                          in_bias=in_bias if biased else None, sums=rows is sums)
        x = rows.bfloat16().double() + (in_bias.double() if biased else 0.0)
        for r, (start, end) in enumerate(zip(starts, starts[1:])):
            slot = len(lengths) - r
            old = before[slot].double()[:reach * channels].view(reach, channels)
            line = torch.cat([old, x[start:end]])
            want = bias.double() + sum(line[j:j + end - start] * weight[:, j].double() for j in range(taps))
            size = bias.double().abs() + sum(line[j:j + end - start].abs() * weight[:, j].double().abs()
                                             for j in range(taps))
            if silu:
                want = torch.nn.functional.silu(want)
            # half a bfloat16 step of the result; the sum's roundings, and those of silu's fast exponential
            assert ((out[start:end] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * (1 + size)).all()
            if reach:
                kept = state[slot].view(-1)[:reach * channels].view(reach, channels).double()
                assert ((kept - line[-reach:]).abs() <= 2.0 ** -24 * line[-reach:].abs()).all()
        assert torch.equal(state[0], before[0])


@pytest.mark.parametrize("layout,heads,rank,rot,dims,row", [
    (0, 3, 32, 64, 64, 96), (1, 5, 64, 64, 32, 160), (0, 2, 16, 24, 8, 48), (1, 33, 192, 64, 64, 256),
])
def test_latent_queries_in_pieces(layout, heads, rank, rot, dims, row):
    """Rows that begin on 16 bytes against ones that do not, which go one coordinate at a time."""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(heads)
    tokens, offset = 5, 8 * heads
    wide = torch.randn(tokens, offset + heads * rot + 9, device="cuda").bfloat16()
    width = offset + heads * rot
    positions = torch.tensor([0, 1, 77, 2047, 5000], dtype=torch.int32, device="cuda")
    exact = 10000.0 ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)
    outs = []
    for shift in (0, 1):
        q = torch.empty(tokens, width + 8 - width % 8 + shift, device="cuda").bfloat16()
        q[:, shift:shift + width] = wide[:, :width]
        q = q[:, shift:]
        out = torch.full((tokens, heads * row), 3.0, device="cuda").bfloat16()
        ops.latent_queries(q, offset, out, positions, exact.float().cuda(), exact.cuda(), dims, layout, tokens,
                           heads, rank, rot, row, amplitude=1.25)
        outs.append(out.view(tokens, heads, row).float())
    pieces, single = outs
    assert (pieces[..., :rank] == 3.0).all() and (pieces[..., rank + rot:] == 0.0).all()
    # the same two products and their sum: at most one rounding apart
    assert ((pieces - single).abs() <= 2.0 ** -7 * single.abs() + 1e-6).all()
    assert torch.equal(pieces[..., rank + dims:], single[..., rank + dims:])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("clear", [False, True])
def test_gated_activation_in_fours(dtype, clear):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(1)
    tokens, width = 300, 4100      # more numbers than threads of the resident CTAs
    values = torch.randn(tokens, 2 * width, device="cuda") * 4
    acts = []
    for pad in (4, 5):             # rows on 16 bytes, and rows that are not
        rows = torch.full((tokens, 2 * width + pad), 9.0, device="cuda")
        rows[:, :2 * width] = values
        act = torch.zeros(tokens, width, dtype=dtype, device="cuda")
        ops.swiglu(rows[:, :2 * width], act, zero_input=clear)
        assert (rows[:, 2 * width:] == 9.0).all()
        assert (rows[:, :2 * width] == 0.0).all() if clear else torch.equal(rows[:, :2 * width], values)
        acts.append(act)
    assert torch.equal(*acts)
