"""What a parameter change and a tuning run capture beside their steps (wd_debug_graph_captures).

Steps are CUDA graphs, captured when first needed and dropped when dt, a contact parameter,
the skin or the contact kernel changes. On lists each of the two buffer parities has a step
graph with three launchers of builds, and two graphs for a build that the host asks for; runs
that are long enough add the chains, 14 remainders and 2 chains of eight steps."""
from __future__ import annotations

import ctypes

import pytest

from test_gpu_auto_lists import _touching
from test_gpu_lists import _same
from world_b200 import ParticleDynamics
from world_b200._lib import check, lib
from world_b200.scenes import column_collapse

pytestmark = pytest.mark.gpu


def _captures(sim):
    got = ctypes.c_int64()
    check(lib.wd_debug_graph_captures(sim.handle, ctypes.byref(got)))
    return got.value


@pytest.mark.parametrize("skin", [0.0, 0.5e-3])
def test_a_changed_parameter_costs_step_graphs_only(skin):
    cfg, st, rad = _touching(71, True)
    cfg.kernel_timing = False
    cfg.neighbor_skin = skin
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    ref.set_neighbor_skin(0.0)
    for s in (sim, ref):
        s.advance(300)
    assert _captures(sim) >= 16                 # chains among them
    for k in range(4):
        before = _captures(sim)
        for s in (sim, ref):
            if k % 2:
                s.dt = 1e-5 * (1 - 1e-3 * k)
            else:
                s.set_contact_params(0.5 - 0.01 * (k + 1), 0.5, 1e5)
            s.advance(40)
        assert _captures(sim) - before <= 12
        _same(ref, sim)
    before = _captures(sim)
    for s in (sim, ref):
        s.advance(300)
    assert _captures(sim) - before >= 16        # long runs at one setting have chains again
    _same(ref, sim)


@pytest.mark.parametrize("steps", [20, 150])
def test_autotune_captures_no_chains(steps):
    """The tuner times every candidate stepping one by one: its captures are the candidates'
    step graphs and builds, made by the untimed steps before (36 list candidates of at most
    12 graphs, the searched step and the first ones), and no chains of steps, which a timed
    run would capture between its two events."""
    sc = column_collapse(4096, diameters="uniform", mu=0.5, cic=32)
    sc.cfg.kernel_timing = False
    ref = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
    sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
    sim.autotune(steps=steps)
    assert _captures(sim) <= 43 * 12
    for s in (ref, sim):
        s.advance(300)
    _same(ref, sim)


def test_autotune_has_one_searched_candidate():
    """Grains that cross half of any skin within a step or two: searching wins. Its kernel has
    a block of its own, so the block reported beside it is always the same."""
    cfg, st, rad = _touching(72, False)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3] += 150.0
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    for _ in range(6):
        assert sim.autotune(steps=10) == (0.0, 256)
    assert sim.tuning()["contact_variant"] == "warp-cooperative"    # lists, if switched on later
