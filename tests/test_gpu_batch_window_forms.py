"""Batched windows on both sides of the rule that packs living slots (short windows of small replicates do not):
every replicate's spectrum equals its plain run's."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import (ConstantModel, Engine, replicate, replicate_mse_pops, replicate_plain_generations)

pytestmark = pytest.mark.gpu


# small replicates below and at the cadence of 26, large ones (over 240 tiles of capacity) at a short cadence
@pytest.mark.parametrize("N0,num_sites,cadence", [(300, 1e7, 7), (300, 1e7, 25), (300, 1e7, 26), (300, 5e9, 5)])
def test_batched_spectra_equal_plain_runs(N0, num_sites, cadence):
    mu = 1e-8
    reps = [replicate(seed1=11 + 2 * r, seed2=501 - 2 * r, num_sites=num_sites, mu=mu, F=0.1 * r, h=0.5,
                      s=ConstantModel.s_from_gamma(-5.0 * r, N0, 0.1 * r) if r else 0.0, N0=N0 + 40 * r, growth_rate=0.002,
                      N_min=100, N_max=2 * N0, num_generations=60 + 13 * r, compact_interval=cadence) for r in range(3)]
    with Engine() as e:
        e.batch_begin(reps)
        e.batch_run()
        got = [e.batch_read_state(r) for r in range(len(reps))]
    for rep, (f, ids, _) in zip(reps, got):
        with Engine() as e:
            e.begin_mse(replicate_mse_pops(rep), seed1=rep.seed1, seed2=rep.seed2, num_sites=rep.num_sites,
                        compact_interval=cadence)
            e.run(replicate_plain_generations(rep))
            want, wid = e.read_state()
        assert np.array_equal(np.ravel(f).view(np.uint32), np.ravel(want).view(np.uint32))
        assert np.array_equal(ids, wid)
