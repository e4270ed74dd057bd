"""Picard steps and their schedule: the right-hand side read between two steps is the last step's,
whether lists have been switched on or off since, and steps whose lists overflow are the searched
ones."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("first", [0.0, 0.4e-3])
def test_rhs_survives_a_switch_of_lists(first, history):
    cfg, st, rad = packed_poly(n=1500, seed=75, mu=0.5, history=history, picard=True)
    cfg.kernel_timing = False
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    cfg.neighbor_skin = first
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    for skin in (0.5e-3, 0.0, 0.3e-3, 0.3e-3, 0.0, 0.0, 0.6e-3):
        for s in (ref, sim):
            s.advance(3)
        np.testing.assert_array_equal(sim.get_rhs(), ref.get_rhs())
        sim.set_neighbor_skin(skin)
        np.testing.assert_array_equal(sim.get_rhs(), ref.get_rhs())
    for s in (ref, sim):
        s.advance(3)
    np.testing.assert_array_equal(sim.get_state(), ref.get_state())
    np.testing.assert_array_equal(sim.get_rhs(), ref.get_rhs())


@pytest.mark.parametrize("kernel", [(128, 64), (256, 48), (256, 0)])
@pytest.mark.parametrize("history", [False, True])
def test_overflowing_lists(kernel, history):
    """Lists of more than 48 entries, and iterates fast enough to change cells within a step."""
    cfg, st, rad = packed_poly(n=1500, seed=76, mu=0.5, history=history, picard=True)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3:] *= 100
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    cfg.neighbor_skin = 1e-2
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_contact_kernel(*kernel)
    for s in (ref, sim):
        s.advance(60)
    assert sim.list_stats()[2] > 40            # the mean: many hold more than 48
    np.testing.assert_array_equal(sim.get_state(), ref.get_state())
    np.testing.assert_array_equal(sim.get_rhs(), ref.get_rhs())
