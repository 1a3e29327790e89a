"""The support mask: the same for every layout of the rows, and without the CUDA library."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import _capi
from parallelpopgen_b200 import surrogate as sg


def _rows():
    p = sg.draw_query_parameters(300, 2)
    p[3, 2], p[4, 5] = np.nan, np.inf
    return p, np.all((p >= sg.LOW) & (p <= sg.HIGH), axis=1)


@pytest.mark.parametrize("built", [True, False])
def test_support_mask(monkeypatch, tmp_path, built):
    if not built:
        monkeypatch.setattr(_capi, "LIB_PATH", tmp_path / "not_built.so")
        monkeypatch.setattr(_capi, "_lib", None)
    p, want = _rows()
    packed = np.zeros(len(p), dtype=np.dtype([("pad", "u1"), ("v", "<f8", 6)]))
    packed["v"] = p
    unaligned = np.frombuffer(b"\0" + p.tobytes(), dtype=np.uint8)[1:].view(np.float64).reshape(p.shape)
    for q in (p, np.asfortranarray(p), p[::-1][::-1], packed["v"], unaligned, p.astype(">f8")):
        got = sg.in_support(q)
        assert got.dtype == bool and np.array_equal(got, want)
    assert sg.in_support(p[:0]).shape == (0,)
