"""The spectrum projection's shapes: every split of the levels into runs, the row itself and its histogram
(frequencies of the device's division, correctly rounded ones, and others), and the batched rows, against
the double-precision CPU projection."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as orc
from parallelpopgen_b200 import ConstantModel, Engine, constant_generations

pytestmark = pytest.mark.gpu

# fp32 output of double sums: half an ulp (6e-8) from the projection, and as much again for the oracle's row
TOL = dict(rtol=2e-7, atol=1e-30)


def _row(seed, M, Nc):
    """Counts of density 1/j with lost and fixed mutations among them; all counts of a small Nc."""
    rng = np.random.default_rng(seed)
    j = np.minimum(np.exp(rng.uniform(0, np.log(Nc), M)).astype(np.int64), Nc - 1)
    j[rng.random(M) < 0.02] = 0
    j[rng.random(M) < 0.02] = Nc
    return j


# runs of 8, 16 and 32 levels: the first and last sample of each shape; rows of one mutation, of part of a
# batch of 32, and (with Nc / 4 < M) histograms
@pytest.mark.parametrize("n", [1, 7, 8, 63, 64, 127, 128, 255, 256, 511, 512, 1000, 1023, 1024, 2047])
@pytest.mark.parametrize("M", [1, 31, 33, 2000])
def test_projection_shapes(n, M):
    Nc = 4096
    row = (_row(n + M, M, Nc) / np.float32(Nc)).astype(np.float32)
    with Engine() as e:
        got = e.site_frequency_spectrum(row, Nc, n, 1e6).astype(np.float64)
    np.testing.assert_allclose(got, orc.sfs(row, n, 1e6), **TOL)


@pytest.mark.parametrize("Nc", [30, 20_000, 400_000])
@pytest.mark.parametrize("kind", ["rounded", "off grid"])
def test_projection_of_host_rows(Nc, kind):
    """A histogram (M > Nc / 4) of correctly rounded quotients, and one that the row replaces because some
    frequency is on neither grid."""
    j = _row(Nc, Nc // 2 + 100, Nc)
    row = j.astype(np.float32) / np.float32(Nc)
    if kind == "off grid":
        row[len(row) // 2] = np.nextafter(np.float32(0.3), np.float32(1)) if Nc == 30 else np.float32(0.123456789)
    n = min(100, Nc - 1)
    with Engine() as e:
        got = e.site_frequency_spectrum(row, Nc, n, 1e7).astype(np.float64)
    np.testing.assert_allclose(got, orc.sfs(row, n, 1e7), **TOL)


@pytest.mark.parametrize("N,L", [(10_000, 2e7), (300, 2e8)])
def test_projection_of_engine_states(N, L):
    """States of the engine: device quotients, and births of the last generation with the host's 1 / Nchrom_e
    (the row itself at N = 10,000, a histogram at N = 300)."""
    model = ConstantModel(N=N, mu=1e-9 if N > 1000 else 1e-8)
    with Engine() as e:
        e.begin_mse(model.mse_pops(), seed1=3, seed2=4, num_sites=L, compact_interval=25)
        e.run(constant_generations(model, 1, 60, 25))
        f, _ = e.read_state(with_ids=False)
        got = e.site_frequency_spectrum(f[0], model.Nchrom_e, 60, L).astype(np.float64)
    assert f.shape[1] > 500
    np.testing.assert_allclose(got, orc.sfs(f[0], 60, L), **TOL)
