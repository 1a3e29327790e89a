"""Spectra of more replicates than one projection launch takes (its sums are limited to 64 MB): the rows of every
launch equal the spectra of their replicates' states."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import Engine, replicate

pytestmark = pytest.mark.gpu


def test_spectra_of_several_launches():
    n, R, N = 1023, 17_000, 600            # 8,184 rows a launch
    reps = [replicate(seed1=7 + 2 * r, seed2=901 - 2 * r, num_sites=1e5, mu=1e-8, F=0.0, h=0.5, s=0.0, N0=N, N_min=N, N_max=N,
                      num_generations=1, compact_interval=1) for r in range(R)]
    with Engine() as e:
        e.batch_begin(reps)
        e.batch_run()
        got = e.batch_sfs(n, R)
        # 64 MB / (8 bytes x 1,025) = 8,184 rows: the launches' first and last ones
        for r in (0, 1, 8183, 8184, 8185, 16367, 16368, R - 1):
            f, _, _ = e.batch_read_state(r)
            want = e.site_frequency_spectrum(f, 2 * N, n, 1e5)
            np.testing.assert_allclose(got[r].astype(np.float64), want.astype(np.float64), rtol=1e-5, atol=1e-3)
