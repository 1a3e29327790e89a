"""The training step over its dispatch: tile widths of 32, 64 and 128 columns (chosen by the batch), ragged tile
counts and one tile, minibatch rows read in place, and tables that have to be gathered first."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _setup(B, rows, seed):
    from parallelpopgen_b200.surrogate import Mlp, init_params
    rng = np.random.default_rng(seed)
    vec = init_params(seed)
    vec[-99:] = rng.normal(0, 0.1, 99).astype(np.float32)
    x = rng.uniform(-1, 1, (rows, 6)).astype(np.float32)
    t = rng.normal(-4, 1, (rows, 99)).astype(np.float32)

    def net():
        mlp = Mlp(capacity=B, lr=1e-3)
        mlp.set_params(vec)
        return mlp
    return net, vec, x, t


# 148 SMs: 32-wide tiles below 19 row tiles, 64-wide from 19, 128-wide from 37
@pytest.mark.parametrize("B", [128, 1152, 18 * 128, 19 * 128, 36 * 128, 37 * 128, 75 * 128])
def test_gradients_over_tile_widths(B):
    net, vec, x, t = _setup(B, B, B)
    g, loss = net().gradients(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    want, want_loss = mo.gradients(vec, x, t, emulate_bf16=True)
    # same bf16 rounding points; the fp32 accumulation order differs and flips rare bf16 ties
    assert abs(loss - want_loss) < 1e-4 * want_loss
    assert np.linalg.norm(g - want) < 1e-2 * np.linalg.norm(want)


@pytest.mark.parametrize("B", [128, 1152, 19 * 128, 37 * 128])
def test_rows_in_place_equal_gathered_rows(B):
    net, _, x, t = _setup(B, 3 * B + 7, B + 1)
    x, t = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    rows = torch.randint(0, x.shape[0], (2, B), device="cuda", generator=torch.Generator("cuda").manual_seed(B))
    a, b = net(), net()
    la, lb = (torch.zeros(1, device="cuda") for _ in range(2))
    for r in rows:
        xb, tb = x[r].contiguous(), t[r].contiguous()
        torch.cuda.synchronize()
        a.train_step(xb, tb, la.data_ptr())
        b.train_step_rows(x, t, r, lb.data_ptr())
        a.check()
        b.check()
        assert la.item() == lb.item()
    assert np.array_equal(a.get_params(), b.get_params())


def test_training_gathers_tables_it_cannot_read_in_place():
    from parallelpopgen_b200.surrogate import train
    B = 256
    net, _, x, t = _setup(B, 1000, 5)
    x, t = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    xs = torch.empty((1000, 12), device="cuda")[:, ::2]
    ts = torch.empty((99, 1000), device="cuda").T
    xs.copy_(x)
    ts.copy_(t)
    nets = [net(), net()]
    train(nets[0], x, t, steps=3, batch=B, seed=2)
    train(nets[1], xs, ts, steps=3, batch=B, seed=2)
    assert np.array_equal(nets[0].get_params(), nets[1].get_params())
