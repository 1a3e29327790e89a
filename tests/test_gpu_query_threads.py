"""Queries of one surrogate from several host threads: each gets the spectra of its own parameters."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from parallelpopgen_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


def test_threads_get_their_own_spectra():
    mlp = sg.Mlp(capacity=4096)
    mlp.set_params(sg.init_params(3))
    s = sg.Surrogate(mlp, None)
    sizes = (1, 200, 257, 1500, 5000)      # a chunk, a ring, several copying threads, two passes
    params = [sg.draw_parameters(n, n) for n in sizes]
    want = [s.predict(p) for p in params]
    x = torch.from_numpy(sg.encode(params[4][:1280])).cuda()
    y = mlp.forward(x).clone()
    torch.cuda.synchronize()
    wrong, errors = [], []

    def query(k):
        try:
            for _ in range(30):
                if not np.array_equal(s.predict(params[k]), want[k]):
                    wrong.append(sizes[k])
        except Exception as ex:   # noqa: BLE001
            errors.append(ex)

    def forward():
        try:
            for _ in range(100):
                if not torch.equal(mlp.forward(x), y):
                    wrong.append("forward")
        except Exception as ex:   # noqa: BLE001
            errors.append(ex)

    threads = [threading.Thread(target=query, args=(k,)) for k in range(len(sizes))] + [threading.Thread(target=forward)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and not wrong, (errors, wrong)
    mlp.check()


def test_a_training_thread_beside_queries():
    mlp = sg.Mlp(capacity=1024, lr=0.0)     # steps of size zero: the weights stay, the passes are enqueued
    mlp.set_params(sg.init_params(3))
    s = sg.Surrogate(mlp, None)
    p = sg.draw_parameters(300, 1)
    want = s.predict(p)
    g = torch.Generator("cuda").manual_seed(1)
    x, t = torch.rand((1024, 6), device="cuda", generator=g), torch.rand((1024, 99), device="cuda", generator=g)
    torch.cuda.synchronize()
    losses = torch.zeros(200, device="cuda")
    torch.cuda.synchronize()
    wrong = []

    def train():
        for k in range(200):
            mlp.train_step(x, t, losses.data_ptr() + 4 * k)

    def query():
        for _ in range(100):
            if not np.array_equal(s.predict(p), want):
                wrong.append(1)

    threads = [threading.Thread(target=train), threading.Thread(target=query)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    mlp.check()
    assert not wrong and bool((losses == losses[0]).all()) and float(losses[0]) > 0
