"""The float32 product on the tensor cores, at the edges of its tiles, with operands of all sizes and with
ones that are not finite, against double and against the CUDA-core product."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,features,depth,pad", [
    (1, 3, 4, 0), (128, 128, 64, 0), (129, 130, 68, 4), (17, 257, 60, 0), (300, 63, 1000, 8),
    (200, 2500, 132, 0),      # columns of an output row that is no multiple of 16 bytes below
])
def test_every_epilogue(tokens, features, depth, pad):
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens + features)
    x = torch.randn(tokens + 2, depth + pad, device="cuda")[:, :depth]
    w = torch.randn(features, depth + pad, device="cuda")[:, :depth]
    x[1::3] *= 1e30
    x[2::3] *= 1e-30
    x[tokens:] = float("nan")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x[:tokens].double() @ w.double().T
    size = x[:tokens].double().abs() @ w.double().abs().T
    # left out: x1 w2, x2 w1, x2 w2, below 2^-24 of a product together; the 24 sums of a block do not
    # round to nearest (2^-23 each at most), those of the blocks do
    bound = (2.0 ** -24 + 25 * 2.0 ** -23 + (depth // 64 + 1) * 2.0 ** -24) * size
    for width in (features, features + 1):
        out = torch.full((tokens + 2, width), 7.0, device="cuda")
        ops.gemm_split(x, w, out, tokens, ops.EPI_STORE_F32, status)
        assert ((out[:tokens, :features] - want).abs() <= bound).all()
        assert (out[tokens:] == 7.0).all() and (out[:, features:] == 7.0).all()
        again = torch.zeros((tokens, width), device="cuda")
        ops.gemm_split(x, w, again, tokens, ops.EPI_STORE, status)
        assert torch.equal(again[:, :features], out[:tokens, :features])
        added = torch.full((tokens + 2, width), 0.5, device="cuda")
        ops.gemm_split(x, w, added, tokens, ops.EPI_ADD_F32, status)
        assert torch.equal(added[:tokens, :features], out[:tokens, :features] + 0.5)
        assert (added[tokens:] == 0.5).all() and (added[:, features:] == 0.5).all()
    ops.gemm_split(x, w, out, tokens, ops.EPI_STORE_F32, status, softcap=3.0)
    assert ((out[:tokens, :features] - 3.0 * torch.tanh(want / 3.0)).abs() <= bound.clamp(max=6.0) + 1e-6).all()
    assert int(status.item()) == 0


def test_closer_to_64_bits_than_the_chain():
    from helix_runtime_b200.ops import library as ops
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for seed, depth in enumerate((256, 3200, 8640)):
        torch.manual_seed(seed)
        for signs in (torch.randn, torch.rand):
            x, w = signs(130, depth, device="cuda"), signs(200, depth, device="cuda") * 0.02
            out, chain = torch.zeros(130, 200, device="cuda"), torch.zeros(130, 200, device="cuda")
            ops.gemm_split(x, w, out, 130, ops.EPI_STORE_F32, status)
            ops.gemm_simt(x, w, chain, 130, ops.EPI_STORE_F32)
            want = x.double() @ w.double().T
            assert (out - want).norm() <= (chain - want).norm()


def test_what_is_not_finite_is_what_the_chain_says():
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(0)
    x, w = torch.randn(140, 200, device="cuda"), torch.randn(150, 200, device="cuda")
    inf, nan, huge = float("inf"), float("nan"), 3.4e38
    x[3, 7], x[130, 1], x[20, 150], x[21, 0], x[21, 1], x[50] = inf, -inf, nan, inf, -inf, huge
    w[9, 7], w[149, 199], w[30], w[77, 70] = 0.0, inf, 1e-39, -huge
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out, chain = torch.zeros(140, 150, device="cuda"), torch.zeros(140, 150, device="cuda")
    ops.gemm_split(x, w, out, 140, ops.EPI_STORE_F32, status)
    ops.gemm_simt(x, w, chain, 140, ops.EPI_STORE_F32)
    assert int(status.item()) == 0
    assert torch.equal(out.isnan(), chain.isnan())
    odd = ~chain.isfinite() & ~chain.isnan()
    assert odd.any() and torch.equal(out[odd], chain[odd])
    plain = chain.isfinite()
    size = x.double().abs().nan_to_num(0, 0, 0) @ w.double().abs().nan_to_num(0, 0, 0).T
    assert ((out - chain).abs()[plain] <= (201 * 2.0 ** -24 + 26 * 2.0 ** -23) * size[plain]).all()


@pytest.mark.parametrize("small", [1e-34, 1e-36, 1e-38, 1e-39, 3e-44])
def test_small_operands_keep_their_bits(small):
    """The smallest numbers of float32, those without a full mantissa too, beside ones that make ordinary
    sums of them: what float32 holds of an operand all reaches the sum."""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(1)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for swapped in (False, True):
        x, w = torch.randn(140, 68, device="cuda") * small, torch.randn(130, 68, device="cuda") * 1e25
        if swapped:
            x, w = w, x
        tokens, features = x.shape[0], w.shape[0]
        out = torch.zeros(tokens, features, device="cuda")
        ops.gemm_split(x, w, out, tokens, ops.EPI_STORE_F32, status)
        want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
        # the bound of the other operands (see test_every_epilogue)
        assert ((out - want).abs() <= (2.0 ** -24 + 25 * 2.0 ** -23 + 2.0 ** -23) * size).all()
    assert int(status.item()) == 0


def test_which_products_take_it():
    from helix_runtime_b200.ops import library as ops
    x, out = torch.zeros(64, 132, device="cuda"), torch.zeros(64, 20000, device="cuda")
    w = torch.zeros(20000, 132, device="cuda")
    assert ops.gemm_split_takes(x, w, out, 64) and not ops.gemm_split_takes(x, w, out, 16)
    assert not ops.gemm_split_takes(x, w[:64], out, 64)
    assert not ops.gemm_split_takes(x[:, 1:129], w[:, 1:129], out, 64)
    assert not ops.gemm_split_takes(x[:, :130], w[:, :130], out, 64)
    assert not ops.gemm_split_takes(x.bfloat16(), w.bfloat16(), out, 64)


@pytest.mark.parametrize("tokens,features,depth", [
    (129, 129, 68), (256, 128, 64), (257, 300, 132), (300, 63, 4), (520, 9700, 196), (130, 40, 1000),
    (17, 130, 132), (1, 5, 64), (128, 129, 200),
])
def test_pairs_have_the_sums_of_single_tiles(tokens, features, depth):
    """More tokens than a tile, with scratch for their terms and without: the same order of the same sums.
    (9,700 by 520: more tiles than pairs of CTAs.)"""
    from helix_runtime_b200.ops import library as ops
    torch.manual_seed(tokens)
    x, w = torch.randn(tokens, depth + 4, device="cuda")[:, :depth], torch.randn(features, depth, device="cuda")
    x[tokens // 2, 3], w[features // 2, 1] = float("inf"), float("nan")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    size = ops.gemm_split_terms(tokens, depth)
    assert size >= 3 * tokens * depth
    terms = torch.full((size + 64,), float("nan"), dtype=torch.bfloat16, device="cuda")
    for epilogue in (ops.EPI_STORE_F32, ops.EPI_ADD_F32):
        out, plain = torch.full((2, tokens + 1, features + 3), 2.0, device="cuda")
        ops.gemm_split(x, w, out, tokens, epilogue, status, terms=terms[:size])
        ops._check(ops.lib().hx_gemm_split(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), plain.data_ptr(),
                                           plain.stride(0), tokens, features, depth, epilogue, 0.0,
                                           status.data_ptr(), ops._stream()))
        torch.testing.assert_close(out, plain, rtol=0, atol=0, equal_nan=True)
    assert terms[size:].isnan().all() and int(status.item()) == 0


@pytest.mark.parametrize("tokens,features,depth,scratch", [
    (129, 700, 64, 0), (129, 1500, 256, 0), (256, 300, 256, 0), (2048, 16, 64, 0), (100, 300, 128, 0),
    (129, 700, 512, 0), (256, 9000, 64, 0), (512, 4000, 128, 0), (2048, 300, 256, 0),
    (129, 1500, 512, 1), (129, 700, 640, 1), (64, 4000, 256, 1), (512, 9000, 64, 1), (256, 4000, 256, 1),
])
def test_shallow_products_do_not_pay_for_the_cut(tokens, features, depth, scratch):
    """Where the cut of the tokens costs more than it gives the product takes none, and has the bits of the road
    that it takes instead."""
    from helix_runtime_b200.ops import library as ops
    from helix_runtime_b200.parts.base import Workspace
    from helix_runtime_b200.parts.linear import Weight, project
    torch.manual_seed(tokens)
    x, w = torch.randn(tokens, depth, device="cuda"), torch.randn(features, depth, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    workspace = Workspace(torch.device("cuda"))
    out, want = torch.zeros((2, tokens, features), device="cuda")
    project(x, Weight(w), out, tokens, ops.EPI_STORE_F32, status, workspace=workspace)
    assert (workspace.bytes() > 0) == bool(scratch)
    if ops.gemm_split_takes(x, w, out, tokens):
        ops.gemm_split(x, w, want, tokens, ops.EPI_STORE_F32, status, scratch=False)
    else:
        ops.gemm_simt(x, w, want, tokens, ops.EPI_STORE_F32)
    assert torch.equal(out, want) and int(status.item()) == 0
