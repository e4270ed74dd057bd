"""The searched step's force kernel on both sides of its lanes-per-grain rule (32 lanes below
4,096 grains, 8 below 24,576, one from there), and around the contacts its buffers hold (32,
32 and 16 a grain), against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_lists import _roomy
from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


def _check(cfg, st, rad, oracle_for, steps):
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_neighbor_skin(0.0)
    orc = oracle_for(cfg, st, radius=rad)
    sim.advance(steps)
    orc.step(steps)
    assert np.array_equal(sim.get_state(), orc.state)
    assert np.array_equal(sim.get_rhs(), orc.rhs)
    assert sim.history_overflow_count() == orc.hist_overflow
    if cfg.history:
        cnt, part, xi = sim.get_history()
        assert np.array_equal(cnt, orc.hcnt)
        mask = np.arange(24)[None, :] < cnt[:, None]
        assert np.array_equal(part.reshape(-1, 24)[mask], orc.hpart.reshape(-1, 24)[mask])
        assert np.array_equal(xi.reshape(-1, 24, 3)[mask], orc.hxi.reshape(-1, 24, 3)[mask])
    sim.close()


@pytest.mark.parametrize("history,picard", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("n", [1, 33, 4095, 4097, 24575, 24577])
def test_sizes(n, history, picard, oracle_for):
    cfg, st, rad = _roomy(n, 80, 0.5, history, picard)
    _check(cfg, st, rad, oracle_for, 6)


@pytest.mark.parametrize("n", [100, 5000, 25000])
@pytest.mark.parametrize("touching", [15, 16, 17, 31, 32, 33, 60])
def test_many_contacts_on_one_grain(n, touching, oracle_for):
    cfg, _, _ = packed_poly(n=8, seed=81, mu=0.5)
    cfg.physics.gravity = 0.0
    cfg.kernel_timing = False
    L = 0.2
    ph = cfg.physics
    for ax in "xyz":
        setattr(cfg.domain, f"{ax}_min", -L)
        setattr(cfg.domain, f"{ax}_max", L)
        setattr(cfg, f"collision_grid_size_{ax}", 16)
    ph.wall_x_min = ph.wall_y_min = ph.floor_z = -L
    ph.wall_x_max = ph.wall_y_max = ph.ceiling_z = L
    k = np.arange(touching) + 0.5
    z = 1 - 2 * k / touching
    phi = k * np.pi * (1 + 5 ** 0.5)
    unit = np.stack([np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi), z], 1)
    rng = np.random.default_rng(82)
    state = np.zeros((n, 6), np.float32)
    rest = n - touching - 1
    side = int(np.ceil(rest ** (1 / 3)))
    idx = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:rest]
    state[touching + 1:, :3] = -0.19 + idx * 4.5e-3      # 30 grains a side at most: clear of the big one
    state[0, :3] = 0.15
    state[1:touching + 1, :3] = 0.15 + unit * (10e-3 + 1.2e-3 - 1e-5)
    state[:, 3:] = rng.normal(0, 0.1, (n, 3))
    radius = np.full(n, 1.2e-3, np.float32)
    radius[0] = 10e-3
    _check(cfg, state, radius, oracle_for, 12)


@pytest.mark.parametrize("history", [True, False])
@pytest.mark.parametrize("skin,kernel", [(0.0, None), (0.5e-3, (256, 0)), (0.5e-3, (128, 64)), (0.5e-3, (256, 1))])
def test_grains_with_one_nan_coordinate(skin, kernel, history, oracle_for):
    """Grains clear of every wall but for one coordinate that is NaN: that axis' two wall
    forces are the clamp (max(0, min(F, NaN)) = F) added and taken away again, which is NaN
    where there is no clamp and a rounding where there is one. Contacts of the others as ever."""
    for clamp in (0.0, 250.0):                  # 0: no clamp
        cfg, st, rad = _roomy(1500, 83, 0.5, history)
        cfg.physics.max_force = clamp
        cfg.neighbor_skin = skin
        st = st.copy()
        for k, axis in ((100, 0), (700, 1), (1300, 2)):
            st[k, :3] = 1e-3 * (axis - 1)
            st[k, axis] = np.nan
        sim = ParticleDynamics(cfg, state=st, radius=rad)
        if kernel:
            sim.set_contact_kernel(*kernel)
        else:
            sim.set_neighbor_skin(0.0)
        orc = oracle_for(cfg, st, radius=rad)
        sim.advance(3)
        orc.step(3)
        np.testing.assert_array_equal(sim.get_state(), orc.state)
        np.testing.assert_array_equal(sim.get_rhs(), orc.rhs)
        sim.close()
