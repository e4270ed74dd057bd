"""The count of contacts that found no free history slot, on lists: a grain whose contacts a cell
crossing re-ordered is taken up once more, and a Picard step whose iterates left the lists is
redone; the dropped springs of what they replace are not counted."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_lists import _same
from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


def _crowded(small=40):
    """64 large grains centred on corners of cells, each in soft contact with `small` others
    that slide along it and cross into other cells."""
    cfg, _, _ = packed_poly(n=8, seed=51, mu=0.5)
    cfg.kernel_timing = False
    ph = cfg.physics
    ph.gravity = 0.0
    ph.normal_stiffness = 100.0
    for ax in "xyz":
        setattr(cfg.domain, f"{ax}_min", -0.1)
        setattr(cfg.domain, f"{ax}_max", 0.1)
        setattr(cfg, f"collision_grid_size_{ax}", 8)
    ph.wall_x_min = ph.wall_y_min = ph.floor_z = -0.1
    ph.wall_x_max = ph.wall_y_max = ph.ceiling_z = 0.1
    k = np.arange(small) + 0.5
    z = 1 - 2 * k / small
    phi = k * np.pi * (1 + 5 ** 0.5)
    unit = np.stack([np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi), z], 1)
    centre = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.05 - 0.075
    state = np.zeros((64 * (small + 1), 6), np.float32)
    state[:64, :3] = centre
    state[64:, :3] = (centre[:, None] + unit * (11.2e-3 - 4e-4)).reshape(-1, 3)
    spin = np.random.default_rng(1).normal(size=(64 * small, 3))
    state[64:, 3:] = np.cross(np.tile(unit, (64, 1)), spin)
    radius = np.full(len(state), 1.2e-3, np.float32)
    radius[:64] = 10e-3
    return cfg, state, radius


@pytest.mark.parametrize("kernel", [(128, 64), (256, 48), (256, 1), (256, 2), (256, 0)])
def test_dropped_springs_are_counted_once(kernel):
    cfg, st, rad = _crowded()
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    ref.set_neighbor_skin(0.0)
    cfg.neighbor_skin = 0.5e-3
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_contact_kernel(*kernel)
    for _ in range(6):
        for s in (ref, sim):
            s.advance(20)
        assert sim.history_overflow_count() == ref.history_overflow_count()
    assert ref.history_overflow_count() > 1000 and sim.list_resort_count() > 10
    _same(ref, sim)


@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("kernel", [(128, 64), (256, 48), (256, 0)])
def test_redone_picard_steps_count_once(kernel, timing):
    cfg, st, rad = _crowded()
    cfg.kernel_timing = timing
    cfg.time_integrator = "backward_euler_picard"
    cfg.picard_iterations = 3
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    cfg.neighbor_skin = 1e-5
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_contact_kernel(*kernel)
    for _ in range(4):
        for s in (ref, sim):
            s.advance(5)
        assert sim.history_overflow_count() == ref.history_overflow_count()
    assert ref.history_overflow_count() > 1000 and sim.picard_counts()[1] > 0
    _same(ref, sim)
