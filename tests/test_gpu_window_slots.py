"""Windows of small states (a slot per thread, compaction in one launch) and of large ones (a quad per thread
until few slots live, then the living packed) against one launch per generation: the same state bit for
bit, at the sizes where they differ in how they reach it."""
from __future__ import annotations

import numpy as np
import pytest

from parallelpopgen_b200 import ConstantModel, Engine, constant_generations

pytestmark = pytest.mark.gpu


def _state(windows, model, L, gens, ci, start=None):
    with Engine() as e:
        e.set_tuning(windows=windows)
        if start is None:
            e.begin_mse(model.mse_pops(), seed1=11, seed2=12, num_sites=L, compact_interval=ci)
        else:
            e.begin_from_state(*start, seed1=11, seed2=12, num_sites=L, compact_interval=ci)
        e.run(gens)
        f, ids = e.read_state()
        return f.copy(), ids.copy(), e.stats()


def _same(model, L, gens, ci, start=None):
    (fa, ia, sa), (fb, ib, sb) = (_state(w, model, L, gens, ci, start) for w in (1, 0))
    assert fa.shape == fb.shape
    assert np.array_equal(fa.view(np.uint32), fb.view(np.uint32))
    assert np.array_equal(ia, ib)
    assert (sa["mutation_generations"], sa["generations"], sa["compactions"]) == (
        sb["mutation_generations"], sb["generations"], sb["compactions"])
    return fa.shape[1]


# windows of one generation, of the longest kind (128) and past it; states of a few slots (tails of every
# length), of several blocks, and past the line to the packing kernel (about 600,000 slots), there also with
# every draw on the binomial search (Nchrom_e below 100)
@pytest.mark.parametrize("N,L,ngen,ci,gamma,F,h", [
    (40, 2e5, 37, 1, 0.0, 0.0, 0.5), (500, 3e5, 60, 7, -20.0, 0.3, 0.1), (2000, 1e6, 300, 130, 5.0, 0.0, 1.0),
    (1000, 1e4, 100, 25, 0.0, 0.0, 0.5), (10_000, 2e7, 130, 25, -10.0, 0.2, 0.5), (10_000, 7e8, 40, 20, 0.0, 0.0, 0.5),
    (10_000, 1.1e9, 30, 15, -3.0, 0.0, 0.2), (10_000, 3e9, 57, 27, 4.0, 0.1, 0.9), (40, 6e10, 45, 20, 0.0, 0.0, 0.5)])
def test_slot_windows_equal_generations(N, L, ngen, ci, gamma, F, h):
    s = ConstantModel.s_from_gamma(gamma, N, F) if gamma else 0.0
    model = ConstantModel(N=N, mu=1e-8 if N < 5000 else 1e-9, s=s, F=F, h=h)
    _same(model, L, constant_generations(model, 1, ngen, ci), ci)


def test_slot_windows_from_states_with_preserved_lost_and_fixed_slots():
    """A resumed state holding preserved, lost (both zeros), fixed and ordinary slots, an extinction in the
    middle of a window, and a window that ends without a compaction."""
    rng = np.random.default_rng(5)
    M, Nc = 1027, 1000
    j = rng.integers(0, Nc + 1, M)
    j[:100], j[100:140] = 0, Nc
    freq = (j / np.float32(Nc)).astype(np.float32)
    freq[:10] = -0.0
    ids = np.zeros((M, 4), np.int32)
    ids[:, 2] = np.arange(1, M + 1) * np.where(rng.random(M) < 0.2, -1, 1)
    model = ConstantModel(N=Nc // 2, mu=1e-8)
    gens = constant_generations(model, 1, 53, 10, final_generation=-1)
    assert _same(model, 1e6, gens, 10, (freq, ids)) > 200
    dead = gens.copy()
    pop = dead["pop"][:, 0]
    pop["Nchrom_e"][24:], pop["alive"][24:], pop["mutate"][24:] = 0, 0, 0
    assert _same(model, 1e6, dead, 10, (freq, ids)) > 100      # the preserved slots stay


def test_infinite_coefficient_keeps_lost_slots_drawn():
    """With an infinite dominance coefficient the selected frequency of a lost slot is not a number, which the
    generation kernel draws from; a window may not take the slot as lost for good."""
    model = ConstantModel(N=200, mu=1e-8, s=0.01)
    gens = constant_generations(model, 1, 20, 10)
    gens["pop"]["h"][5, 0] = np.inf
    _same(model, 1e6, gens, 10)
