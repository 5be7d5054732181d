"""Products of prompt portions by pairs of CTAs (tiles of 256 tokens): every epilogue at the edges of
the tiles, with row-major and tiled weights, against double."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    # tokens, features, depth
    (129, 256, 64), (255, 300, 72), (256, 128, 200), (257, 1000, 1000), (511, 64, 448),
    (700, 9000, 136),        # more tiles than pairs: both accumulators are used again
    (2300, 1300, 64),        # the second half of the last tile is empty
    (250, 20000, 72),        # 79 tiles of 256 columns: a round, then five tiles in four pieces each
    (1200, 4800, 200),       # 95: a round, then 21 in halves; 38 pairs of 128 up and gate columns
    (140, 3000, 64),         # no whole round: every tile in pieces
    (300, 2250, 4096),       # sums: every tile in pieces
    (1500, 3400, 4096),      # sums: a round of whole tiles, then pieces
]


@pytest.mark.parametrize("tiled", [False, True])
@pytest.mark.parametrize("tokens,features,depth", SHAPES)
def test_every_epilogue(tokens, features, depth, tiled):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens + features)
    x = (torch.randn(tokens + 5, depth) * 0.5).bfloat16().cuda()
    x[tokens:] = float("nan")
    rows = -(-features // 128) * 128 if tiled else features      # the up rows start on a tile
    w = (torch.randn(rows + features, depth) * 0.1).bfloat16().cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    held = ops.tile_weights(w) if tiled else w
    options = dict(weight_shape=tuple(w.shape)) if tiled else {}
    want = x[:tokens].double() @ w.double().T
    size = x[:tokens].double().abs() @ w.double().abs().T
    # float32 sums of `depth` products, in any order
    bound = (depth + 2) * 2.0 ** -24 * size
    gate, up = want[:, :features], want[:, rows:rows + features]
    out = torch.full((tokens + 2, features), 7.0, device="cuda")
    ops.gemm_tc(x, held, out, tokens, features, ops.EPI_STORE_F32, status, **options)
    assert ((out[:tokens] - gate).abs() <= bound[:, :features]).all() and (out[tokens:] == 7.0).all()
    out = torch.full((tokens + 2, features + 4), 0.5, device="cuda")
    ops.gemm_tc(x, held, out, tokens, features, ops.EPI_ADD_F32, status, **options)
    assert ((out[:tokens, :features] - 0.5 - gate).abs()
            <= bound[:, :features] + 2.0 ** -22).all()
    assert (out[tokens:] == 0.5).all() and (out[:, features:] == 0.5).all()
    out = torch.full((tokens + 2, features), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc(x, held, out, tokens, features, ops.EPI_STORE, status, **options)
    assert ((out[:tokens].double() - gate).abs() <= 2.0 ** -8 * gate.abs() + bound[:, :features]).all()
    assert (out[tokens:] == 7.0).all()
    ops.gemm_tc(x, held, out, tokens, features, ops.EPI_SWIGLU, status, up_row_offset=rows, **options)
    act = torch.nn.functional.silu(gate) * up
    slack = (1.1 * up.abs() + 1e-3) * bound[:, :features] + gate.abs() * bound[:, rows:rows + features]
    assert ((out[:tokens].double() - act).abs()
            <= (2.0 ** -8 + 2.0 ** -18) * act.abs() + 2 * slack + 1e-6).all()
    assert (out[tokens:] == 7.0).all()
    assert int(status.item()) == 0


def test_an_ordered_sum_repeats_bit_for_bit():
    """Sizes whose last round of tiles is shared out by atomic adds unless the caller wants an order."""
    from helix_runtime_b200.ops import library as ops
    from helix_runtime_b200.parts.linear import Weight, project
    torch.manual_seed(3)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for tokens, features, depth in ((512, 4096, 4096), (1200, 4096, 4096), (300, 2050, 11008)):
        x = torch.randn(tokens, depth, device="cuda").bfloat16()
        matrix = torch.randn(features, depth, device="cuda").bfloat16()
        before = torch.randn(tokens, features, device="cuda")
        want = before.double() + x.double() @ matrix.double().T
        for weight in (Weight(matrix), Weight(matrix, tile=False)):
            first = None
            for _ in range(40):
                out = before.clone()
                project(x, weight, out, tokens, ops.EPI_ADD_F32, status, True)
                first = out if first is None else first
                assert torch.equal(out, first)
            size = before.double().abs() + x.double().abs() @ matrix.double().abs().T
            assert ((first - want).abs() <= (depth + 2) * 2.0 ** -24 * size).all()
    assert int(status.item()) == 0
