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
