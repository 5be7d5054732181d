"""Stored products of few tiles, whose CTAs share a tile's depth as a cluster, at the edges of tiles and runs."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,features,depth", [
    (1, 16, 4096), (16, 130, 2048), (17, 128, 2056), (33, 300, 2120), (64, 1280, 4096), (65, 16, 2048),
    (100, 257, 3096), (128, 24, 2776), (129, 16, 4096), (300, 1280, 2048), (2048, 16, 4096), (1, 4096, 4096),
    (1, 7500, 2048), (5, 16, 2040),      # the most tiles, and a depth below the rule's
])
def test_clusters_add_up_their_parts(tokens, features, depth):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens + features)
    x = torch.randn(tokens + 3, depth + 8, device="cuda").bfloat16()[:, :depth]
    w = torch.randn(features, depth, device="cuda").bfloat16()
    x[tokens:] = float("nan")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x[:tokens].double() @ w.double().T
    size = x[:tokens].double().abs() @ w.double().abs().T
    # float32 sums of at most depth products, cut off or rounded at every step: 2^-23 each of the running sum
    bound = (depth // 16 + 32) * 2.0 ** -23 * size
    for weights, shape in ((w, None), (ops.tile_weights(w), (features, depth))):
        for epilogue, dtype in ((ops.EPI_STORE_F32, torch.float32), (ops.EPI_STORE, torch.bfloat16)):
            outs = []
            for _ in range(2):
                out = torch.full((tokens + 2, features + 5), 7.0, dtype=dtype, device="cuda")
                ops.gemm_tc(x, weights, out, tokens, features, epilogue, status, weight_shape=shape)
                outs.append(out)
            rounding = 2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0.0
            assert ((outs[0][:tokens, :features] - want).abs() <= bound + rounding).all()
            assert (outs[0][tokens:] == 7.0).all() and (outs[0][:, features:] == 7.0).all()
            assert torch.equal(*outs)      # one order of the sums
    out = torch.zeros(tokens, features, device="cuda")
    ops.gemm_tc(x, w, out, tokens, features, ops.EPI_STORE_F32, status, softcap=5.0)
    assert ((out - 5.0 * torch.tanh(want / 5.0)).abs() <= bound + 1e-5).all()
    assert int(status.item()) == 0


@pytest.mark.parametrize("tokens,features,depth,cut", [
    (129, 16, 2048, 0), (300, 512, 2560, 0), (1500, 16, 2048, 0), (2048, 100, 3008, 0), (700, 256, 2048, 0),
    (129, 16, 3072, 1), (1500, 16, 4096, 1), (2048, 100, 6144, 1), (128, 16, 2048, 1),
])
def test_shallow_prompts_keep_one_chain(tokens, features, depth, cut):
    """More than 128 tokens of a depth below 3,072 are faster as one chain over the depth: the bits of a sum
    that is added up by one writer, which is never cut."""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens)
    x = torch.randn(tokens, depth, device="cuda").bfloat16()
    w = torch.randn(features, depth, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, chain = torch.zeros((2, tokens, features), device="cuda")
    ops.gemm_tc(x, w, out, tokens, features, ops.EPI_STORE_F32, status)
    ops.gemm_tc(x, w, chain, tokens, features, ops.EPI_ADD_F32, status, ordered=True)
    assert torch.equal(out, chain) == (not cut) and int(status.item()) == 0


@pytest.mark.parametrize("features,depth", [(16, 4096), (300, 2120), (1280, 8192)])
def test_ordered_products_do_not_depend_on_the_number_of_tokens(features, depth):
    """One token, a weight stream, a prompt's few tiles and many: the same bits of a token's sums, through the
    entry that every layer uses."""
    from helix_runtime_b200.ops import library as ops
    from helix_runtime_b200.parts.linear import Weight, project
    torch.manual_seed(features)
    x = torch.randn(700, depth, device="cuda").bfloat16()
    w = Weight(torch.randn(features, depth, device="cuda").bfloat16())
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for epilogue, dtype in ((ops.EPI_STORE_F32, torch.float32), (ops.EPI_STORE, torch.bfloat16)):
        for softcap in (0.0, 30.0) if epilogue == ops.EPI_STORE_F32 else (0.0,):
            want = torch.zeros(700, features, dtype=dtype, device="cuda")
            project(x, w, want, 700, epilogue, status, ordered=True, softcap=softcap)
            for tokens in (1, 16, 17, 64, 100, 128, 129, 300):
                out = torch.zeros(tokens, features, dtype=dtype, device="cuda")
                project(x, w, out, tokens, epilogue, status, ordered=True, softcap=softcap)
                assert torch.equal(out, want[:tokens])
    assert int(status.item()) == 0
