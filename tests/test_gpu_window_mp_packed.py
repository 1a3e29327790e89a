"""Multi-population windows in their two forms -- small blocks with a slot per thread, and half tiles that pack
their living slots -- against one launch per generation: sizes on both sides of the line between them, records
under which a lost mutation need not stay lost, and a window end that leaves a half tile empty."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import Engine

from test_gpu_window_mp import assert_same, mse_start, run_both
from test_gpu_window_mp import schedule as schedule_four


def schedule(P, *args, **kw):
    """The schedule with inbreeding and dominance for eight populations."""
    return schedule_four(P, *args, F=(0.0, 0.0, 0.2, 0.1, 0.0, 0.3, 0.0, 0.1),
                         h=(0.5, 0.3, 0.5, 0.8, 0.1, 0.6, 0.5, 0.0), **kw)


pytestmark = pytest.mark.gpu


# a window ends with under 600,000 slots at the two smaller sizes, with a million and more at the largest
@pytest.mark.parametrize("P", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("num_sites", [2e5, 2e7, 1.5e8])
def test_windows_of_every_size(P, num_sites):
    gens = schedule(P, 1, 110, found=(0, 1, 10), compact_interval=25, sample_every=60)
    out = run_both(lambda e: e.begin_mse(mse_start(P), seed1=7, seed2=8, num_sites=num_sites, compact_interval=25),
                   [gens])
    l1, l0 = assert_same(out, min_slots=100)
    assert l1 < l0 / 3


@pytest.mark.parametrize("num_sites", [2e6, 1.5e8])
@pytest.mark.parametrize("odd", ["selection", "migration"])
def test_lost_mutations_that_need_not_stay_lost(num_sites, odd):
    """An infinite coefficient makes the selected frequency of a lost mutation, or its migration sum, not a
    number: no slot may be taken for lost for good."""
    gens = schedule(3, 1, 60, found=(0, 1, 2), sample_every=10**6)
    if odd == "selection":
        gens["pop"][20:24, 1]["sel_intercept"] = np.inf
    else:
        gens["migration"][20, 0] = np.inf
    out = run_both(lambda e: e.begin_mse(mse_start(3), seed1=9, seed2=10, num_sites=num_sites, compact_interval=25),
                   [gens])
    assert_same(out, min_slots=100)


@pytest.mark.parametrize("M", [1, 3, 127, 128, 129, 511, 512, 513, 1024, 1025, 700_000, 700_416 + 513])
def test_resumed_states_of_edge_sizes(M):
    rng = np.random.default_rng(M)
    N = 4000
    freq = rng.integers(0, N, size=(2, M)).astype(np.float32) / np.float32(N)
    freq[:, rng.random(M) < 0.3] = 0
    freq[0, 0] = 0.5
    ids = np.zeros((M, 4), dtype=np.int32)
    ids[:, 2] = np.arange(1, M + 1)
    gens = schedule(2, 1, 40, found=(0, 1), sizes=(2000, 2000), mu=0.0, compact_interval=17)
    out = run_both(lambda e: e.begin_from_state(freq, ids, seed1=1, seed2=2, num_sites=2e6, compact_interval=17), [gens])
    assert_same(out, min_slots=0 if M < 200 else M // 8)


@pytest.mark.parametrize("P", [4, 5, 8])
def test_windows_at_their_length_limit(P):
    """128 generations up to four populations, 64 above; without compactions a window ends there."""
    gens = schedule(P, 1, 200, compact_interval=0, sample_every=10**6)
    gens["compact"] = 0
    gens["preserve"] = 0
    out = run_both(lambda e: e.begin_mse(mse_start(P), seed1=3, seed2=4, num_sites=3e5, compact_interval=0), [gens])
    assert_same(out, min_slots=100)
