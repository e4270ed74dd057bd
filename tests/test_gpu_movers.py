"""The mover sort at the edges of its caps (8,192 movers below 2^16 grains, 16,384 below 2^19,
28,672 from there) and of its rounds (one mover per warp up to 4,704, four above): the
order after thousands of grains changed cell is the (cell key, grain id) order."""
from __future__ import annotations

import numpy as np
import pytest

from world_b200 import ParticleDynamics, SimConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,moved,radix", [(65535, 8192, False), (65535, 8193, True), (65536, 8193, False),
                                           (70000, 4704, False), (70000, 4705, False), (70000, 1, False),
                                           (70000, 16384, False), (70000, 16385, True),
                                           (524287, 16385, True), (524288, 28672, False),
                                           (524288, 28673, True), (524288, 0, False)])
def test_order_after_many_moves(n, moved, radix):
    cells = 128
    cfg = SimConfig()
    for ax in "xyz":
        setattr(cfg.domain, f"{ax}_min", 0.0)
        setattr(cfg.domain, f"{ax}_max", 1.0)
        setattr(cfg, f"collision_grid_size_{ax}", cells)
    cfg.physics.wall_x_min = cfg.physics.wall_y_min = cfg.physics.floor_z = 0.0
    cfg.physics.particle_radius = 1e-4
    cfg.physics.gravity = 0.0
    cfg.kernel_timing = False
    rng = np.random.default_rng(n + moved)
    cell = rng.integers(1, cells - 1, (n, 3))
    st = np.zeros((n, 6), np.float32)
    st[:, :3] = (cell + 0.5) / cells
    sim = ParticleDynamics(cfg, state=st)
    sim.set_neighbor_skin(0.0)
    sim.advance(1)
    before = sim.radix_search_count()[0]
    who = rng.choice(n, moved, replace=False)
    cell[who] += rng.choice([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, 0, -1], [1, 1, 1]], moved) if moved else 0
    st[:, :3] = (cell + 0.5) / cells
    sim.set_state(st)
    keys = (cell[:, 0] * cells + cell[:, 1]) * cells + cell[:, 2]
    skeys, sids = sim.debug_sorted()
    order = np.lexsort((np.arange(n), keys))
    np.testing.assert_array_equal(sids, order)
    np.testing.assert_array_equal(skeys, keys[order])
    assert (sim.radix_search_count()[0] > before) == radix
    sim.close()
