"""A device-side graph launch that fails (a list build, or the radix path of a search) leaves
its step undone. The next call that waits reports it, once: after list steps, searched steps,
batches and reads alike. wd_debug_launch_failure notes the failure; no launch fails here."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_auto_lists import _touching
from test_gpu_lists import _same
from world_b200 import ParticleDynamics, SceneBatch, WorldError
from world_b200._lib import check, lib, ptr
from world_b200.scenes import column_collapse

pytestmark = pytest.mark.gpu


def _reported_once(sim, work):
    work()
    sim.synchronize()
    check(lib.wd_debug_launch_failure(sim.handle))
    work()
    with pytest.raises(WorldError, match="device-side graph launch failed"):
        sim.synchronize()
    work()
    sim.synchronize()


@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("skin", [0.0, 0.5e-3])
def test_steps_report_a_failed_launch(skin, history):
    cfg, st, rad = _touching(91, history)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_neighbor_skin(skin)
    _reported_once(sim, lambda: sim.advance(2))
    ref.advance(6)
    np.testing.assert_array_equal(sim.get_state(), ref.get_state())


def test_a_searched_batch_reports_a_failed_launch():
    members = [column_collapse(n, diameters="uniform", mu=0.5, cic=16) for n in (512, 1024)]
    for m in members:
        m.cfg.kernel_timing = False
    batch = SceneBatch.from_scenes(members)
    _reported_once(batch, lambda: batch.advance(2))


def test_reads_report_a_failed_launch_of_a_searched_step():
    cfg, st, rad = _touching(92, False)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_neighbor_skin(0.0)
    for read in (sim.get_state, sim.compute_momentum, sim.compute_total_energy):
        sim.advance(3)
        check(lib.wd_debug_launch_failure(sim.handle))
        with pytest.raises(WorldError, match="device-side graph launch failed"):
            read()
        read()


@pytest.mark.parametrize("asynchronous", [False, True])
@pytest.mark.parametrize("skin", [0.0, 0.5e-3])
def test_a_handle_recovers_with_an_upload(skin, asynchronous):
    """Steps after a lost one leave nothing to rely on: an upload starts from the order of the
    grain ids and without springs, as a new handle does."""
    cfg, st, rad = _touching(93, True)
    cfg.kernel_timing = False
    cfg.neighbor_skin = skin
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_neighbor_skin(skin)
    sim.advance(200)
    assert sim.get_history()[0].sum() > 0
    check(lib.wd_debug_launch_failure(sim.handle))
    with pytest.raises(WorldError, match="device-side graph launch failed"):
        sim.synchronize()
    if asynchronous:
        check(lib.wd_set_state_async(sim.handle, ptr(st)))
        sim.synchronize()
    else:
        sim.set_state(st)
    assert sim.get_history()[0].sum() == 0
    fresh = ParticleDynamics(cfg, state=st, radius=rad)
    for s in (sim, fresh):
        s.advance(60)
    _same(fresh, sim)
