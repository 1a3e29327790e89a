"""A host query whose forward pass gave up a bounded wait (an accumulator hand-off withheld by the test) reports it
once instead of returning what the buffers held, and the next query is exact."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import GoFishError, _capi
from parallelpopgen_b200 import surrogate as sg

pytestmark = pytest.mark.gpu

DEVICE_FAULT = next(k for k, v in _capi.STATUS_NAMES.items() if v == "GF_ERR_DEVICE")


# one chunk, several, and two passes of the network's capacity; the fused kernel and one GEMM per layer
@pytest.mark.parametrize("rows", [1, 256, 257, 700])
@pytest.mark.parametrize("fused", [1, 0])
def test_query_reports_a_withheld_hand_off(rows, fused):
    mlp = sg.Mlp(capacity=512)
    mlp.set_params(sg.init_params(3))
    assert mlp.lib.gf_mlp_set_fused_inference(mlp.h, fused) == 0
    s = sg.Surrogate(mlp, None)
    p = sg.draw_parameters(rows, rows)
    want = s.predict(p)
    assert mlp.lib.gf_mlp_inject_fault(mlp.h, 1) == 0
    with pytest.raises(GoFishError) as err:
        s.predict(p)
    assert err.value.status == DEVICE_FAULT
    assert np.array_equal(s.predict(p), want)     # reported once, cleared
    mlp.check()
