"""Products added to a float32 output: the edges of the tiles and of the 32 columns that a warp takes, rows
and outputs that are not 16-byte aligned, against double."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("tokens,features,depth,row,offset", [
    (129, 256, 64, 256, 0), (160, 257, 72, 260, 0), (255, 287, 200, 288, 4), (300, 289, 64, 289, 0),
    (257, 1030, 1000, 1036, 1), (700, 9001, 136, 9004, 0), (1500, 3403, 4096, 3403, 3), (2300, 1300, 64, 1302, 0),
])
def test_sums_onto_an_output(tokens, features, depth, row, offset, ordered):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens + features)
    x = torch.randn(tokens, depth, device="cuda").bfloat16()
    w = torch.randn(features, depth, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    memory = torch.randn(offset + (tokens + 2) * row, device="cuda")
    before = memory.clone()
    old, out = (m[offset:].view(tokens + 2, row) for m in (before, memory))
    ops.gemm_tc(x, w, out, tokens, features, ops.EPI_ADD_F32, status, ordered=ordered)
    product = x.double() @ w.double().T
    # float32 sums of `depth` products and the old value, in any order
    size = x.double().abs() @ w.double().abs().T + old[:tokens, :features].double().abs()
    assert ((out[:tokens, :features].double() - old[:tokens, :features].double() - product).abs()
            <= (depth + 2) * 2.0 ** -24 * size).all()
    assert torch.equal(out[tokens:], old[tokens:]) and torch.equal(out[:, features:], old[:, features:])
    assert torch.equal(memory[:offset], before[:offset]) and int(status.item()) == 0
