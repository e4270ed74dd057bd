"""Energies of stored springs where the search sorts all keys: more grains have changed cells
since the last search than the mover path takes, as in a handle's first search and after an
upload. The springs' counts are kept in the order of the state's slots, which that path has to
tell the energy as the other one does."""
from __future__ import annotations

import numpy as np
import pytest

from scale_cases import transplant
from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics, SceneBatch

pytestmark = pytest.mark.gpu

N = 16385                                      # above the 8,192 movers of scenes this small


def _springs():
    cfg, st, rad = packed_poly(n=N, seed=71, mu=0.5)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.advance(40)
    state, springs = sim.get_state().reshape(-1, 6).copy(), sim.get_history()
    sim.close()
    return cfg, state, rad, springs


def test_first_search_and_upload(oracle_for):
    cfg, state, rad, springs = _springs()
    assert springs[0].sum() > 10000
    sim = ParticleDynamics(cfg, state=state, radius=rad)
    sim.set_history(*springs)
    expect = transplant(sim, oracle_for).energy()
    radix = sim.radix_search_count()[0]
    assert sim.compute_total_energy() == pytest.approx(expect, rel=1e-12)
    assert sim.radix_search_count()[0] == radix + 1
    assert sim.grain_energies().sum() == pytest.approx(expect, rel=1e-12)
    sim.advance(5)
    mirrored = sim.get_state().reshape(-1, 6).copy()
    mirrored[:, :6] *= -1                       # nearly every grain in another cell
    sim.set_state(mirrored)
    expect = transplant(sim, oracle_for).energy()
    radix = sim.radix_search_count()[0]
    assert sim.compute_total_energy() == pytest.approx(expect, rel=1e-12)
    assert sim.radix_search_count()[0] == radix + 1


def test_batch(oracle_for):
    cfg, state, rad, springs = _springs()
    alone = ParticleDynamics(cfg, state=state, radius=rad)
    alone.set_history(*springs)
    batch = SceneBatch([cfg, cfg], [state, state], radii=[rad, rad])
    count, partner, xi = springs
    batch.set_history(np.concatenate([count] * 2), np.concatenate([partner] + [np.where(partner >= 0, partner + N, partner)]),
                      np.concatenate([xi] * 2))
    expect = transplant(alone, oracle_for).energy()
    np.testing.assert_allclose(batch.scene_energies(), [expect, expect], rtol=1e-12)
