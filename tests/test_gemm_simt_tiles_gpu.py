"""The CUDA-core product in every tile it has: at the edges of the tiles, with rows that do not
begin on 16 bytes, and with the promise that a sum does not depend on the tile it falls into."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("features,depth,pad", [
    (150, 70, 0),            # few tiles: the small ones for every number of tokens
    (9500, 36, 0),           # 149 tiles of 64 features
    (19000, 33, 1),          # 149 tiles of 128; no row but the first begins on 16 bytes
])
def test_every_tile_gives_the_same_sums(features, depth, pad, dtype):
    from helix_runtime_b200.ops import library as ops
    rng = np.random.default_rng(features)
    most = 130
    make = lambda rows: torch.tensor(rng.normal(size=(rows, depth + pad)), dtype=torch.float32) \
        .to(dtype).cuda()[:, :depth]
    x, w = make(most), make(features)
    want = x.double() @ w.double().T
    # every term is rounded once at most and every addition once: (depth + 1) half units in the
    # last place of the sum of magnitudes
    bound = (depth + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    whole = None
    for tokens in (most, 129, 65, 64, 33, 32, 17, 16, 5, 4, 1):
        out = torch.full((most, features), 7.0, device="cuda")
        ops.gemm_simt(x, w, out, tokens, ops.EPI_STORE_F32)
        assert ((out[:tokens] - want[:tokens]).abs() <= bound[:tokens]).all()
        assert (out[tokens:] == 7.0).all()
        whole = out if whole is None else whole
        assert torch.equal(out[:tokens], whole[:tokens])
        added = torch.full((most, features), 0.5, device="cuda")
        ops.gemm_simt(x, w, added, tokens, ops.EPI_ADD_F32)
        assert torch.equal(added[:tokens], whole[:tokens] + 0.5)
        stored = torch.zeros((most, features), dtype=dtype, device="cuda")
        ops.gemm_simt(x, w, stored, tokens, ops.EPI_STORE)
        assert torch.equal(stored[:tokens], whole[:tokens].to(dtype))
