"""Products of a few float32 tokens: tiles that hang over tokens, features and depth, several tiles a CTA, every
epilogue, padded rows, against double; and a value does not depend on the call's other rows."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("features,depth,padding", [(64, 256, 0), (5, 1001, 3), (993, 259, 1), (3202, 1000, 4),
                                                    (4740, 516, 0), (17281, 300, 0)])
@pytest.mark.parametrize("tokens", [1, 2, 3, 5, 8, 9, 16, 17, 31, 40, 128])
def test_products_of_few_tokens(tokens, features, depth, padding):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens + features)
    x = torch.randn(tokens + 1, depth + padding, device="cuda")
    w = torch.randn(features + 1, depth + padding, device="cuda")
    x[tokens], w[features] = float("nan"), float("nan")
    x[:, depth:], w[:, depth:] = float("nan"), float("nan")
    x, w = x[:, :depth], w[:features, :depth]
    out = torch.full((tokens + 2, features + 3), 0.5, device="cuda")
    if not ops.gemm_few_takes(x, w, out, tokens):
        assert tokens > 16
        with pytest.raises(RuntimeError):
            ops.gemm_few(x, w, out, tokens, ops.EPI_STORE_F32)
        return
    want = x[:tokens].double() @ w.double().T
    # float32 sums of `depth` products, in any order, and one more addition
    bound = (depth + 2) * 2.0 ** -24 * (x[:tokens].double().abs() @ w.double().abs().T + 0.5)
    ops.gemm_few(x, w, out, tokens, ops.EPI_ADD_F32)
    assert ((out[:tokens, :features] - 0.5 - want).abs() <= bound).all()
    assert (out[tokens:] == 0.5).all() and (out[:, features:] == 0.5).all()
    ops.gemm_few(x, w, out, tokens, ops.EPI_STORE_F32)
    assert ((out[:tokens, :features] - want).abs() <= bound).all()
    alone = torch.empty((1, features), device="cuda")
    ops.gemm_few(x[tokens - 1:], w, alone, 1, ops.EPI_STORE)      # (every row begins on 16 bytes)
    assert torch.equal(alone[0], out[tokens - 1, :features])
    ops.gemm_few(x, w, out, tokens, ops.EPI_STORE_F32, softcap=30.0)
    # tanh has a slope of one at most; its own float32 error is a few units of 30
    assert ((out[:tokens, :features] - 30.0 * torch.tanh(want / 30.0)).abs() <= bound + 30.0 * 2.0 ** -21).all()
    assert (out[tokens:] == 0.5).all() and (out[:, features:] == 0.5).all()
