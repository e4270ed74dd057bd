"""Other work on the device, on the default stream, while a handle is set up and steps: nothing
of the handle's waits behind it and lands later, on top of what its own stream has done since."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_auto_lists import _touching
from test_gpu_lists import _same
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu

HALF_A_SECOND = 1_000_000_000      # clock cycles


@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("skin", [0.0, 0.2e-3])
def test_steps_beside_a_busy_default_stream(skin, history):
    """Grains that cross half the skin every few steps, so that most builds fall inside chains."""
    cfg, st, rad = _touching(95, history)
    cfg.kernel_timing = False
    st = st.copy()
    st[:, 3:] = np.random.default_rng(96).normal(0, 1.0, (2744, 3))
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    ref.set_neighbor_skin(0.0)
    cfg.neighbor_skin = skin
    # the kernels' first use loads them, which waits for the device
    with ParticleDynamics(cfg, state=st, radius=rad) as warm:
        warm.advance(200)
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    torch.cuda._sleep(HALF_A_SECOND)
    busy = torch.cuda.Event()
    busy.record()
    sim.advance(200)
    sim.synchronize()
    assert not busy.query()
    torch.cuda.synchronize()
    for _ in range(3):
        sim.advance(200)
    ref.advance(800)
    _same(ref, sim)
    assert sim.time == ref.time


def test_a_handle_is_whole_when_it_is_there():
    """Nothing of a handle's creation is still to come when the call returns."""
    cfg, st, rad = _touching(97, True)
    cfg.kernel_timing = False
    ref = ParticleDynamics(cfg, state=st, radius=rad)
    ref.advance(3)
    torch.cuda._sleep(HALF_A_SECOND)
    busy = torch.cuda.Event()
    busy.record()
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.advance(3)
    sim.synchronize()
    assert not busy.query()
    torch.cuda.synchronize()
    _same(ref, sim)


def test_an_uploaded_tensor_is_read_before_its_memory_is_reused():
    """The upload is queued behind other work on the handle's stream, and the tensor (here also
    the contiguous copy that the call makes) is gone when the call returns."""
    cfg, st, rad = _touching(98, False)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.set_state(-st)
    stream = torch.cuda.ExternalStream(sim.stream_ptr())
    by_column = torch.from_numpy(st).cuda().t().contiguous().t()
    assert not by_column.is_contiguous()

    def reuse():
        out = [torch.full_like(by_column, 7.0, memory_format=torch.contiguous_format) for _ in range(4)]
        torch.cuda.current_stream().synchronize()
        return out

    reuse()                                    # the kernels' first use loads them, which waits
    sim.set_state_tensor(by_column * 1.0)
    sim.set_state(-st)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(HALF_A_SECOND)
    busy = torch.cuda.Event()
    busy.record(stream)
    sim.set_state_tensor(by_column)
    sim.set_state_tensor(by_column * 1.0)
    others = reuse()
    assert not busy.query()
    sim.synchronize()
    del others
    np.testing.assert_array_equal(sim.get_state().reshape(-1, 6), st)


@pytest.mark.parametrize("own", [False, True])
def test_a_read_waits_for_work_queued_on_its_memory(own):
    """The tensor that takes the state, the caller's or a new one, has memory that torch still
    writes to or reads from."""
    cfg, st, rad = _touching(99, False)
    cfg.kernel_timing = False
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.synchronize()
    out = torch.zeros(6 * sim.n, device="cuda")
    seen = torch.empty_like(out)
    seen.copy_(out)
    torch.cuda.synchronize()
    torch.cuda._sleep(HALF_A_SECOND)
    if own:
        out.fill_(7.0)
        got = sim.state_tensor(out)
    else:
        seen.copy_(out)
        del out
        got = sim.state_tensor()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got.cpu().numpy().reshape(-1, 6), st)
    assert own or not seen.any()


@pytest.mark.parametrize("wait", [False, True])
def test_an_uploaded_tensor_may_outlive_the_handle(wait):
    cfg, st, rad = _touching(99, False)
    cfg.kernel_timing = False
    kept = torch.from_numpy(st).cuda()
    for _ in range(3):
        sim = ParticleDynamics(cfg, state=st, radius=rad)
        sim.set_state_tensor(kept)
        sim.set_state_tensor(kept * 1.0)
        if wait:
            sim.synchronize()
        sim.close()
    del kept
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
