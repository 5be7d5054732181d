"""Grouped products of many tokens, a group's rows cut into equal tiles of up to 256: lists with runs of
every length, against double."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs,rows,features,depth", [
    ([(0, 1)], 128, 128, 64),
    # (group, entries of 32 rows): a tile of every size, two, and three; none of group 1; no rows behind
    ([(2, 1), (0, 2), (3, 3), (2, 4), (0, 5), (3, 6), (0, 7), (2, 8), (3, 9), (0, 17), (-1, 3)], 304, 300, 200),
    ([(1, 40), (-1, 33), (3, 64), (0, 31)], 1040, 1030, 72),      # more units than pairs of CTAs
    ([(g % 4, 1) for g in range(70)], 48, 40, 136),               # a tile an entry
    ([(-1, 5)], 64, 64, 64),
])
def test_runs_of_every_length(runs, rows, features, depth):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(rows + len(runs))
    listed = [group for group, entries in runs for _ in range(entries)]
    tokens, groups = 32 * len(listed), 4
    x = (torch.randn(tokens, depth) * 0.5).bfloat16().cuda()
    for entry, group in enumerate(listed):
        if group < 0:
            x[32 * entry:32 * entry + 32] = float("nan")
    w = (torch.randn(groups, 2 * rows, depth) * 0.1).bfloat16().cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tile_group = torch.tensor(listed, dtype=torch.int32).cuda()
    out = torch.full((tokens, features + 2), 7.0, device="cuda")
    act = torch.full((tokens, features + 2), 7.0, dtype=torch.bfloat16, device="cuda")
    assert ops.gemm_tc_runs_supports(tokens, w, rows) and ops.gemm_tc_runs_supports(tokens, w, 0)
    ops.gemm_tc_runs(x, w, out, tokens, features, tile_group, status)
    ops.gemm_tc_runs(x, w, act, tokens, features, tile_group, status, rows, ops.GATE_SILU)
    assert int(status.item()) == 0
    assert (out[:, features:] == 7.0).all() and (act[:, features:] == 7.0).all()
    for entry, group in enumerate(listed):
        part = slice(32 * entry, 32 * entry + 32)
        if group < 0:
            assert (out[part] == 7.0).all() and (act[part] == 7.0).all()
            continue
        gate = x[part].double() @ w[group, :features].double().T
        up = x[part].double() @ w[group, rows:rows + features].double().T
        # float32 sums of `depth` products, in any order
        bound = (depth + 2) * 2.0 ** -24 * (x[part].double().abs() @ w[group].double().abs().max(0)[0][:, None])
        assert ((out[part, :features] - gate).abs() <= bound).all()
        want = torch.nn.functional.silu(gate) * up
        assert ((act[part, :features].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -18) * want.abs()
                + 2 * bound * (1.1 * up.abs() + gate.abs() + 1e-3) + 1e-6).all()


@pytest.mark.parametrize("token_tile", [16, 32, 64, 128, 256])
def test_tiles_of_every_size_the_grouped_product_takes(token_tile):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(token_tile)
    listed, rows, features, depth = [2, -1, 0], 144, 136, 200
    tokens = token_tile * len(listed)
    x = (torch.randn(tokens, depth) * 0.5).bfloat16().cuda()
    w = (torch.randn(3, 2 * rows, depth) * 0.1).bfloat16().cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    tile_group = torch.tensor(listed, dtype=torch.int32).cuda()
    out = torch.full((tokens, features), 7.0, device="cuda")
    act = torch.full((tokens, features), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tc_grouped(x, w, out, tokens, features, ops.EPI_STORE_F32, 0, token_tile, tile_group, status)
    ops.gemm_tc_grouped(x, w, act, tokens, features, ops.EPI_SWIGLU, rows, token_tile, tile_group, status)
    assert int(status.item()) == 0
    for tile, group in enumerate(listed):
        part = slice(token_tile * tile, token_tile * (tile + 1))
        if group < 0:
            assert (out[part] == 7.0).all() and (act[part] == 7.0).all()
            continue
        gate = x[part].double() @ w[group, :features].double().T
        up = x[part].double() @ w[group, rows:rows + features].double().T
        # as in test_runs_of_every_length
        bound = (depth + 2) * 2.0 ** -24 * (x[part].double().abs() @ w[group].double().abs().max(0)[0][:, None])
        assert ((out[part] - gate).abs() <= bound).all()
        want = torch.nn.functional.silu(gate) * up
        assert ((act[part].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -18) * want.abs()
                + 2 * bound * (1.1 * up.abs() + gate.abs() + 1e-3) + 1e-6).all()


def test_sizes_that_take_another_road():
    from helix_runtime_b200.ops import library as ops
    supports = ops.lib().hx_gemm_tc_runs_supports
    assert supports(32 * 4096, 16, 96, 48, 64, 64) and not supports(32 * 4097, 16, 96, 48, 64, 64)
    assert not supports(48, 16, 96, 48, 64, 64) and not supports(64, 16, 96, 48, 60, 64)
    assert not supports(64, 16, 96, 40, 64, 64) and supports(64, 16, 88, 0, 64, 64)
