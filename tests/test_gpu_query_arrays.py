"""Mlp.predict reads whole rows of doubles from the caller's array, whatever its type and layout; other shapes are
refused."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


def test_predict_takes_any_array_of_rows():
    mlp = sg.Mlp(capacity=128)
    mlp.set_params(sg.init_params(3))
    scaling = sg.Surrogate(mlp, None)._scaling()
    p = sg.draw_parameters(100, 1).astype(np.float32)
    want = mlp.predict(p.astype(np.float64), scaling)
    wide = np.zeros((100, 12))
    wide[:, ::2] = p
    for q in (p, np.asfortranarray(p), wide[:, ::2], p.astype(">f8"), p.tolist()):
        assert np.array_equal(mlp.predict(q, scaling), want)
    for q in (p[:, :5], p[0], np.zeros((2, 3, 6))):
        with pytest.raises(ValueError):
            mlp.predict(q, scaling)
