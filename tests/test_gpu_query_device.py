"""Surrogate queries answered on the device from the parameters to the normalised spectra: the same network
outputs through the host's own encoding and normalisation, at the edges of tiles, chunks and passes, with and
without a target scale, and the calls that take the general path."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import surrogate as sg

pytestmark = pytest.mark.gpu


def _surrogate(capacity, scaled=True):
    mlp = sg.Mlp(capacity=capacity)
    mlp.set_params(sg.init_params(3))
    k = np.arange(1, 100)
    rng = np.random.default_rng(4)
    scale = sg.TargetScale(-np.log(k) - 1.7, 0.3 + 0.3 * rng.uniform(size=99)) if scaled else None
    return sg.Surrogate(mlp, None, scale=scale)


# one row; a tile and one more; a chunk (256 rows) and its neighbours; two and four copying threads; a pass (the network's
# capacity, at most 8,192 rows) and its neighbours; several passes
@pytest.mark.parametrize("capacity,rows", [(128, 1), (128, 128), (128, 129), (4096, 255), (4096, 256), (4096, 257),
                                           (4096, 2049), (4096, 4096), (4096, 4097), (16_384, 8192), (16_384, 16_385)])
@pytest.mark.parametrize("scaled", [True, False])
def test_queries_equal_the_host_path(capacity, rows, scaled):
    s = _surrogate(capacity, scaled)
    p = sg.draw_parameters(rows, rows)
    p[0] = sg.LOW
    p[-1] = sg.HIGH
    got, routed = s.query(p)
    want = s._predict_arrays(p)
    assert got.shape == (rows, 99) and got.dtype == np.float64 and not routed.any()
    # double throughout: exponents up to ~10 of size, one rounding each (2^-53), an exp and a sum of 99
    np.testing.assert_allclose(got, want, rtol=1e-13)


def test_other_calls_take_the_general_path():
    s = _surrogate(256)
    p = sg.draw_parameters(200, 1)
    want = s.predict(p)
    assert np.array_equal(s.predict(np.asfortranarray(p)), want)
    assert np.array_equal(s.predict(np.repeat(p, 2, axis=0)[::2]), want)
    assert np.array_equal(s.predict(p.tolist()), want)
    assert s.predict(p[:0]).shape == (0, 99)
    assert np.array_equal(s.query(p[7])[0], s.predict(p[7:8]))
    with pytest.raises((ValueError, IndexError)):
        s.predict(p[:, :5])
    s.scale = sg.TargetScale(s.scale.mean[:98], s.scale.std[:98])
    with pytest.raises(ValueError):
        s.predict(p)


def test_support_mask():
    p = sg.draw_query_parameters(500, 2)
    p[3, 2], p[4, 5] = np.nan, np.inf
    p[5], p[6] = sg.LOW, sg.HIGH
    want = np.all((p >= sg.LOW) & (p <= sg.HIGH), axis=1)
    assert want.any() and not want.all() and want[5] and want[6] and not want[3] and not want[4]
    for q in (p, np.asfortranarray(p), p.astype(np.float32).astype(np.float64)[:, :]):
        ok = sg.in_support(q)
        assert ok.dtype == bool
    assert np.array_equal(sg.in_support(p), want) and np.array_equal(sg.in_support(np.asfortranarray(p)), want)
