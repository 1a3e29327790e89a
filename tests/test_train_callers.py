"""Which networks and tables a training run reads in place: everything else takes train_step on gathered rows."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from parallelpopgen_b200 import surrogate as sg


class _Recorder:
    """A network of the caller's own: the methods that train() has always used."""

    def __init__(self):
        self.batches = []

    def set_learning_rate(self, lr):
        pass

    def train_step(self, x, t, d_loss=None):
        self.batches.append((x.clone(), t.clone()))

    def check(self):
        pass


def test_another_network_gets_gathered_rows(monkeypatch):
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    x = torch.arange(40 * 6, dtype=torch.float32).reshape(40, 6)
    t = torch.arange(40 * 99, dtype=torch.float32).reshape(40, 99)
    net = _Recorder()
    sg.train(net, x, t, steps=3, batch=8, seed=5, log_every=0)
    assert len(net.batches) == 3
    for xb, tb in net.batches:
        rows = (xb[:, 0] / 6).long()
        assert torch.equal(xb, x[rows]) and torch.equal(tb, t[rows])


@pytest.mark.gpu
def test_tables_read_in_place():
    mlp = sg.Mlp(capacity=128)
    x, t = torch.zeros((300, 6), device="cuda"), torch.zeros((300, 99), device="cuda")
    assert sg._reads_rows_in_place(mlp, x, t)
    assert not sg._reads_rows_in_place(_Recorder(), x, t)
    assert not sg._reads_rows_in_place(mlp, x.double(), t)
    assert not sg._reads_rows_in_place(mlp, x.t().contiguous().t(), t)
    assert not sg._reads_rows_in_place(mlp, x, t[:299])
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):      # the indices would be drawn on a stream that the network does not wait for
        assert not sg._reads_rows_in_place(mlp, x, t)
        assert sg._reads_rows_in_place(sg.Mlp(capacity=128, stream=side.cuda_stream), x, t)
    with pytest.raises(ValueError):
        mlp.train_step_rows(x, t, torch.zeros(128, dtype=torch.int32, device="cuda"))


@pytest.mark.gpu
def test_tables_that_need_gradients_are_refused():
    mlp = sg.Mlp(capacity=128)
    x, t = torch.zeros((300, 6), device="cuda", requires_grad=True), torch.zeros((300, 99), device="cuda")
    with pytest.raises(RuntimeError):
        sg.train(mlp, x, t, steps=1, batch=128)


@pytest.mark.gpu
def test_a_network_on_its_own_stream_trains_alike():
    g = torch.Generator("cuda").manual_seed(1)
    x = torch.rand((300, 6), device="cuda", generator=g) * 2 - 1
    t = torch.rand((300, 99), device="cuda", generator=g)
    weights = []
    for side in (None, torch.cuda.Stream()):
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            mlp = sg.Mlp(capacity=128, stream=side.cuda_stream if side else None)
            mlp.set_params(sg.init_params(2))
            sg.train(mlp, x, t, steps=4, batch=128, seed=3, log_every=0)
            weights.append(mlp.get_params())
    assert np.array_equal(weights[0], weights[1])
