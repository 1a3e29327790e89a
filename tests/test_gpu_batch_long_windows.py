"""Batched windows longer than the generation records a block stages (128): every replicate equals its plain run,
with the records resident and built per super-step."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import (ConstantModel, Engine, replicate, replicate_mse_pops, replicate_plain_generations)

pytestmark = pytest.mark.gpu


def _replicates(cadences, N0, num_sites):
    return [replicate(seed1=31 + 2 * r, seed2=707 - 2 * r, num_sites=num_sites, mu=1e-8, F=0.1 * (r % 3), h=0.5,
                      s=ConstantModel.s_from_gamma(-4.0 * r, N0, 0.1 * (r % 3)) if r else 0.0, N0=N0 + 30 * r,
                      growth_rate=0.001, N_min=100, N_max=2 * N0, num_generations=2 * cadence + 37 + r,
                      compact_interval=cadence) for r, cadence in enumerate(cadences)]


# one cadence at the limit, past it, past a block's threads; long and short ones together; several tiles
@pytest.mark.parametrize("cadences,N0,num_sites", [
    ((128, 128), 300, 1e7), ((129, 129), 300, 1e7), ((200, 200), 300, 1e7), ((300, 257), 300, 1e7),
    ((10, 129, 300, 25), 300, 1e7), ((130, 64), 2000, 5e7)])
@pytest.mark.parametrize("budget", [1 << 26, 0])
def test_long_windows_equal_plain_runs(cadences, N0, num_sites, budget):
    reps = _replicates(cadences, N0, num_sites)
    with Engine() as e:
        e.batch_set_record_budget(budget)
        e.batch_begin(reps)
        e.batch_run()
        got = [e.batch_read_state(r) for r in range(len(reps))]
    for rep, (f, ids, gen) in zip(reps, got):
        assert gen == rep.num_generations
        with Engine() as e:
            e.begin_mse(replicate_mse_pops(rep), seed1=rep.seed1, seed2=rep.seed2, num_sites=rep.num_sites,
                        compact_interval=rep.compact_interval)
            e.run(replicate_plain_generations(rep))
            want, wid = e.read_state()
        assert np.array_equal(np.ravel(f).view(np.uint32), np.ravel(want).view(np.uint32))
        assert np.array_equal(ids, wid)
