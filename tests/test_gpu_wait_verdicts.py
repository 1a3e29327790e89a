"""A hand-off withheld by the test at batches of one tile to several rounds over the device: every warp of every
CTA leaves its waits together, the fault is reported once, and the next pass is exact."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from parallelpopgen_b200 import surrogate as sg

pytestmark = pytest.mark.gpu

GF_ERR_DEVICE = 6


# an odd CTA without rows, one tile of a pair, a device's worth and one more, three rounds
@pytest.mark.parametrize("tiles", [1, 2, 3, 148, 149, 375])
@pytest.mark.parametrize("fused", [1, 0])
def test_withheld_hand_off_ends_every_wait(tiles, fused):
    B = 128 * tiles
    mlp = sg.Mlp(capacity=B)
    mlp.set_params(sg.init_params(tiles))
    assert mlp.lib.gf_mlp_set_fused_inference(mlp.h, fused) == 0
    g = torch.Generator("cuda").manual_seed(tiles)
    x = torch.rand((B, 6), device="cuda", generator=g) * 2 - 1
    t = torch.rand((B, 99), device="cuda", generator=g)
    want = mlp.forward(x).cpu().numpy()
    mlp.check()
    for _ in range(2):
        assert mlp.lib.gf_mlp_inject_fault(mlp.h, 1) == 0
        mlp.forward(x)
        assert mlp.lib.gf_mlp_check(mlp.h) == GF_ERR_DEVICE
        assert mlp.lib.gf_mlp_check(mlp.h) == 0
        assert np.array_equal(mlp.forward(x).cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert np.isfinite(mlp.gradients(x, t)[1])    # a training pass afterwards finds its waits as they were
    mlp.check()
