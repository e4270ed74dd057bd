"""A tuning run leaves the handle where it was: state, springs, counts, and the right-hand side of
the last step, which the trial steps overwrite."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_lists import _same
from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("picard", [False, True])
@pytest.mark.parametrize("skin", [0.0, 0.4e-3])
def test_the_last_step_survives_tuning(skin, picard):
    cfg, st, rad = packed_poly(n=1500, seed=77, mu=0.5, picard=picard)
    cfg.kernel_timing = False
    cfg.particles_per_cell = 2
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    cfg.neighbor_skin = skin
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    for _ in range(3):
        for s in (ref, sim):
            s.advance(5)
        counts = sim.grid_overflow_count(), sim.history_overflow_count(), sim.list_stats()[0]
        sim.autotune(steps=4)
        assert counts == (sim.grid_overflow_count(), sim.history_overflow_count(), sim.list_stats()[0])
        np.testing.assert_array_equal(sim.get_rhs(), ref.get_rhs())
        assert sim.compute_max_acceleration() == ref.compute_max_acceleration()
        _same(ref, sim)
