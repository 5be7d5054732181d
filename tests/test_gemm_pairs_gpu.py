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


@pytest.mark.parametrize("tile_groups,rows,features,depth", [
    ([2, 0, 0, 1, -1], 300, 150, 200),       # a group of two tiles, one without tokens at the end
    ([0], 256, 128, 64),
    ([3, 1, 1, 0, 2, 2, 2, -1, -1, -1, -1], 2100, 1000, 72),      # more tiles than pairs
])
def test_groups_of_whole_tiles(tile_groups, rows, features, depth):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(rows)
    tokens, groups = 256 * len(tile_groups), 4
    x = (torch.randn(tokens, depth) * 0.5).bfloat16().cuda()
    w = (torch.randn(groups, 2 * rows, depth) * 0.1).bfloat16().cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    listed = torch.tensor(tile_groups, dtype=torch.int32).cuda()
    out = torch.full((tokens, features), 7.0, device="cuda")
    act = torch.full((tokens, features), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc_grouped(x, w, out, tokens, features, ops.EPI_STORE_F32, 0, 256, listed, status)
    ops.gemm_tc_grouped(x, w, act, tokens, features, ops.EPI_SWIGLU, rows, 256, listed, status)
    assert int(status.item()) == 0
    for tile, group in enumerate(tile_groups):
        part = slice(256 * tile, 256 * tile + 256)
        if group < 0:
            assert (out[part] == 7.0).all() and (act[part] == 7.0).all()
            continue
        gate = x[part].double() @ w[group, :features].double().T
        up = x[part].double() @ w[group, rows:rows + features].double().T
        size = x[part].double().abs() @ w[group].double().abs().max(0)[0][:, None]
        bound = (depth + 2) * 2.0 ** -24 * size
        assert ((out[part] - gate).abs() <= bound).all()
        want = torch.nn.functional.silu(gate) * up
        assert ((act[part].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -18) * want.abs()
                + 2 * bound * (1.1 * up.abs() + gate.abs() + 1e-3) + 1e-6).all()
