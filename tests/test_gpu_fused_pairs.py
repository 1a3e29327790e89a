"""The fused forward on pairs of CTAs at batches whose tiles do not pair up: odd tile counts, with and without rows
of the network's capacity behind them, and one to three rounds over the device."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,capacity_tiles", [(1, 1), (1, 2), (2, 2), (3, 3), (3, 8), (147, 147), (148, 148), (149, 149),
                                                  (297, 300), (375, 375)])
def test_pairs_equal_layers(tiles, capacity_tiles):
    from parallelpopgen_b200.surrogate import Mlp, init_params
    mlp = Mlp(capacity=128 * capacity_tiles)
    vec = init_params(tiles)
    vec[-99:] = np.random.default_rng(tiles).normal(0, 0.1, 99).astype(np.float32)
    mlp.set_params(vec)
    B = 128 * tiles
    g = torch.Generator("cuda").manual_seed(tiles)
    if capacity_tiles > tiles:   # leaves other rows behind the batch
        mlp.forward(torch.rand((128 * capacity_tiles, 6), device="cuda", generator=g) * 2 - 1)
    x = torch.rand((B, 6), device="cuda", generator=g) * 2 - 1
    out = torch.full((B + 256, 99), 7.25, device="cuda")
    torch.cuda.synchronize()
    mlp.forward_ptr(x.data_ptr(), B, out.data_ptr())
    mlp.check()
    assert bool((out[B:] == 7.25).all())          # nothing behind the batch is written
    assert mlp.lib.gf_mlp_set_fused_inference(mlp.h, 0) == 0
    want = mlp.forward(x)
    mlp.check()
    assert torch.equal(out[:B].view(torch.int32), want.view(torch.int32))
