"""The reverse pass ends where the window did: state, springs, the last step's right-hand side
and largest acceleration are those of the forward pass, whichever schedule it took, and the
steps after it go on from there."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_auto_lists import _touching
from test_gpu_lists import _same
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,every", [(8, 8), (40, 20), (11, 4)])
@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("schedule", ["searched", "own lists", "lists"])
def test_backward_leaves_the_window_s_end(schedule, history, steps, every):
    cfg, st, rad = _touching(98, history)
    cfg.kernel_timing = False
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    ref.set_neighbor_skin(0.0)
    cfg.neighbor_skin = 0.3e-3 if schedule == "lists" else 0.0
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    if schedule == "searched":
        sim.set_neighbor_skin(0.0)
    for s in (ref, sim):
        s.advance(60)
    ref.advance(steps)
    sim.adjoint_record(steps, every)
    assert (sim.kernels_per_step() >= 5) == (schedule == "searched")
    rhs = sim.get_rhs()
    g = torch.from_numpy(np.random.default_rng(99).normal(size=(2744, 3)).astype(np.float32)).cuda()
    sim.adjoint_backward(g, 1e-3 * g)
    np.testing.assert_array_equal(sim.get_rhs(), rhs)
    assert sim.compute_max_acceleration() == ref.compute_max_acceleration()
    _same(ref, sim)
    for s in (ref, sim):
        s.advance(20)
    _same(ref, sim)
