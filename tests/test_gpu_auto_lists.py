"""simulation.neighbor_skin 0: the library searches every step, or steps on lists of its
own choice where a run of steps pays for them. Either way the results are the searched
step's to the last bit: states, springs, rhs, energies and the lifetime count of
overfull cells. The searched side is a handle on which set_neighbor_skin(0) was called,
which always searches."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import OracleSim, params_from_config
from test_gpu_lists import _same
from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics, SimConfig
from world_b200.state_io import grain_properties, initial_state

pytestmark = pytest.mark.gpu


def _both(cfg, state, radius=None):
    own = ParticleDynamics(cfg, state=state, radius=radius)
    searched = ParticleDynamics(cfg, state=state, radius=radius)
    searched.set_neighbor_skin(0.0)
    return own, searched


def _equal(own, searched):
    assert own.grid_overflow_count() == searched.grid_overflow_count()
    assert own.history_overflow_count() == searched.history_overflow_count()
    _same(searched, own)
    assert own.list_stats()[0] == 0 and own.tuning()["neighbor_skin_m"] == 0.0


def _touching(seed, history):
    """Equal grains a percent of their diameter apart, flying at 0.3 m/s: contacts soon and
    everywhere, but no grain fast enough to leave its neighbours within a few steps."""
    cfg, st, rad = packed_poly(n=2744, seed=seed, history=history)
    d = 5e-3
    idx = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    st[:, :3] = (idx - 6.5) * 1.01 * d + rng.uniform(-0.004 * d, 0.004 * d, (2744, 3))
    st[:, 3:] = rng.normal(0, 0.3, (2744, 3))
    return cfg, st, np.full(2744, 0.5 * d, np.float32)


@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("history", [False, True])
def test_runs_between_uploads_of_many_lengths(history, timing):
    cfg, st, rad = _touching(61, history)
    cfg.kernel_timing = timing
    own, searched = _both(cfg, st, rad)
    for run in (1, 1, 5, 6, 7, 40, 2, 3, 100, 13, 1):
        for sim in (own, searched):
            sim.advance(run)
        _equal(own, searched)
        state = own.get_state()
        for sim in (own, searched):
            sim.set_state(state)
    for _ in range(30):
        for sim in (own, searched):
            sim.take_step()
    assert own.kernels_per_step() == 2          # it did step on lists
    _equal(own, searched)
    for sim in (own, searched):
        sim.dt = 0.5e-5
        sim.advance(20)
    _equal(own, searched)


@pytest.mark.parametrize("ppc", [0, 1, 2, 3, 4])
def test_overfull_cells_are_counted_at_every_step(ppc, oracle_for):
    """particles_per_cell around the packing's occupancy: the count, taken after every
    step, equals the oracle's, which searches each step's starting state."""
    cfg, st, rad = packed_poly(n=2500, seed=62, mu=0.3)
    cfg.particles_per_cell = ppc
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3:] *= 8
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    orc = oracle_for(cfg, st, radius=rad)
    sim.advance(8)
    orc.step(8)
    for _ in range(40):
        sim.take_step()
        orc.step()
        assert sim.grid_overflow_count() == orc.overflow
    sim.advance(200)
    orc.step(200)
    assert sim.grid_overflow_count() == orc.overflow
    assert np.array_equal(sim.get_state(), orc.state)


def test_a_fast_flow_goes_back_to_searching():
    """Grains that cross half a skin every step or two: lists would build all the time."""
    cfg, st, rad = packed_poly(n=2500, seed=63, history=False)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3] += 60.0
    own, searched = _both(cfg, st, rad)
    for _ in range(6):
        for sim in (own, searched):
            sim.advance(50)
        _equal(own, searched)
    assert own.kernels_per_step() == 6          # searching again


def test_narrow_cells_are_searched():
    """Cells narrower than a grain: a searched step sees the 27 cells only, so the handle
    must not step on lists (they would hold pairs further apart)."""
    cfg, st, rad = packed_poly(n=2000, seed=64)
    cfg.kernel_timing = False
    for ax in "xyz":
        setattr(cfg, f"collision_grid_size_{ax}", 40)   # 2.5 mm cells, 5 mm grains
    own, searched = _both(cfg, st, rad)
    for sim in (own, searched):
        sim.advance(60)
    _equal(own, searched)
    assert own.kernels_per_step() == 6


def test_default_cube_frames_match_the_oracle(oracle_for):
    cfg = SimConfig()
    cfg.init_jitter = 0.3
    st, _ = initial_state(cfg)
    sim = ParticleDynamics(cfg)
    orc = oracle_for(cfg, st)
    for _ in range(6):
        for _ in range(10):
            sim.take_step()
        orc.step(10)
        sim.unpack_state()
        assert np.array_equal(sim.host_state, orc.state)
        sim.device_state.copy_from_host(sim.host_state)
    assert sim.grid_overflow_count() == orc.overflow
    assert np.array_equal(sim.get_rhs(), orc.rhs)
    t = sim._timings()
    assert t[0] > 0 and t[1] > 0


@pytest.mark.parametrize("steps,every", [(7, 3), (12, 4), (25, 5)])
def test_windows_of_odd_length_give_the_searched_gradient(steps, every):
    torch = pytest.importorskip("torch")
    cfg, st, rad = packed_poly(n=1500, seed=65, mu=0.4)
    cfg.kernel_timing = False
    own, searched = _both(cfg, st, rad)
    g = torch.from_numpy(np.random.default_rng(66).normal(size=(1500, 3)).astype(np.float32)).cuda()
    for _ in range(3):
        out = []
        for sim in (own, searched):
            sim.set_state(st)
            sim.adjoint_record(steps, every)
            gx, gv, th = sim.adjoint_backward(g, 1e-3 * g)
            out.append((sim.get_state(), gx.cpu().numpy(), gv.cpu().numpy(), th))
        for a, b in zip(*out):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("first,kernels", [(36, 6), (37, 2)])
def test_a_new_handle_searches_until_lists_pay(first, kernels):
    """2,744 grains: a call of 36 steps on a new handle is searched, one of 37 is not (40 x
    32768 / (32768 + n) steps, rounded up), and the searched ones count towards the line."""
    cfg, st, rad = _touching(65, True)
    cfg.kernel_timing = False
    own, searched = _both(cfg, st, rad)
    for run, expect in ((first, kernels), (1, 2), (3, 2)):
        for sim in (own, searched):
            sim.advance(run)
        assert own.kernels_per_step() == expect
        _equal(own, searched)


def test_chains_captured_for_both_pairs_of_buffers():
    """A list step swaps the state buffers and the spring rows, a searched one the rows only,
    so a searched step between two long runs changes which of them go together: chains exist
    for both pairings, and the ones captured first still finish their steps after the others
    have been captured. Builds come about every eight steps, most inside chains."""
    cfg, st, rad = _touching(67, True)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3:] = np.random.default_rng(68).normal(0, 1.0, (2744, 3))
    own, searched = _both(cfg, st, rad)
    for run in (200,) + (1, 1, 100) * 5:
        for sim in (own, searched):
            sim.advance(run)
        _equal(own, searched)
        assert own.time == searched.time
        state = own.get_state()
        for sim in (own, searched):
            sim.set_state(state)
    assert own.kernels_per_step() == 2          # the long runs were on lists


def test_the_stage_wait_hook_needs_lists_that_the_caller_asked_for():
    from world_b200 import WorldError
    from world_b200._lib import check, lib
    cfg, st, rad = _touching(69, False)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    for _ in range(2):
        with pytest.raises(WorldError, match="no Verlet lists"):
            check(lib.wd_debug_stage_wait(sim.handle, 0, 0))
        sim.advance(40)
    sim.set_neighbor_skin(0.0)
    with pytest.raises(WorldError, match="no Verlet lists"):
        check(lib.wd_debug_stage_wait(sim.handle, 0, 0))
    sim.set_neighbor_skin(0.5e-3)
    check(lib.wd_debug_stage_wait(sim.handle, 0, 0))


def test_a_rollout_is_queued_without_waiting():
    """A hundred steps are queued behind half a second of other work on the handle's stream:
    the call returns while that work still runs."""
    torch = pytest.importorskip("torch")
    cfg, st, rad = _touching(93, True)
    cfg.kernel_timing = False
    own, searched = _both(cfg, st, rad)
    state = torch.from_numpy(st).cuda()
    stream = torch.cuda.ExternalStream(own.stream_ptr())
    for k in range(4):
        if k == 3:                              # graphs and chains exist by now
            own.synchronize()
            with torch.cuda.stream(stream):
                torch.cuda._sleep(1_000_000_000)
            busy = torch.cuda.Event()
            busy.record(stream)
        for sim in (own, searched) if k < 3 else (own,):
            sim.set_state_tensor(state)
            sim.advance(100)
    assert not busy.query()
    searched.set_state_tensor(state)
    searched.advance(100)
    assert own.kernels_per_step() == 2
    _equal(own, searched)


def test_lists_that_do_not_pay_are_left_within_one_call():
    """One call of 500 steps, nothing read meanwhile: the handle tries lists, learns that
    nearly every step builds, and searches by the end of it."""
    cfg, st, rad = packed_poly(n=2500, seed=63, history=False)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3] += 60.0
    own, searched = _both(cfg, st, rad)
    own.advance(500)
    assert own.kernels_per_step() == 6
    searched.advance(500)
    _equal(own, searched)
