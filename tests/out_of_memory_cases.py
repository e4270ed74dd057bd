"""Calls that find too little device memory: each returns an error, once, and leaves the handle
as it was; with the memory back, the same call gives what it gives on a handle that never ran
short. What was allocated by then is kept and completed, not taken for whole. Run in a process
of its own by test_gpu_out_of_memory.py."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from world_b200 import ParticleDynamics, WorldError
from world_b200._lib import check, lib, ptr
from world_b200.scenes import column_collapse

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once():
    sc = column_collapse(1 << 16, diameters="uniform", mu=0.5, cic=16)
    sc.cfg.neighbor_skin = 0.5e-3              # lists that do not give way
    sc.cfg.kernel_timing = False
    sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
    sim.advance(1)
    before = sim.get_state()
    torch.zeros(1, device="cuda")
    # a window's first checkpoint takes 28 MB
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (10 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(WorldError, match="out of memory"):
        sim.adjoint_record(2, 2)
    np.testing.assert_array_equal(sim.get_state(), before)
    sim.advance(1)
    sim.synchronize()
    del fill
    torch.cuda.empty_cache()
    sim.close()


# bytes left free: too few for the adjoints' spring rows (2 x 12 MB at 2^15 grains), for the
# tape's first, and for its later steps (about 18 MB each)
@pytest.mark.parametrize("left", [10 << 20, 40 << 20, 90 << 20])
def test_a_window_survives_a_failed_allocation(left):
    n, steps, every = 1 << 15, 8, 8
    sc = column_collapse(n, diameters="uniform", mu=0.5, cic=16)
    sc.cfg.neighbor_skin = 0.5e-3              # lists that do not give way
    sc.cfg.kernel_timing = False
    g = torch.from_numpy(np.random.default_rng(94).normal(size=(n, 3)).astype(np.float32)).cuda()
    grid = torch.ones(4 * 16 ** 3, device="cuda")
    out = []
    for short in (False, True):
        sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
        sim.adjoint_record(steps, every)
        if short:
            room = torch.empty((n, 3), device="cuda"), torch.empty((n, 3), device="cuda")
            free = torch.cuda.mem_get_info()[0]
            fill = torch.empty(free - left, dtype=torch.uint8, device="cuda")
            del room
            for _ in range(2):
                with pytest.raises(WorldError, match="out of memory"):
                    sim.adjoint_backward(g, g)
            del fill
            torch.cuda.empty_cache()
        gx, gv, th = sim.adjoint_backward(g, g)
        dx, dv = sim.deposit_vjp(grid)
        out.append([sim.get_state(), th] + [t.cpu().numpy() for t in (gx, gv, dx, dv)])
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("left", [3 << 20, 12 << 20])
def test_lists_for_picard_survive_a_failed_allocation(left):
    sc = column_collapse(1 << 16, diameters="uniform", mu=0.5, cic=16)
    sc.cfg.kernel_timing = False
    sc.cfg.time_integrator = "backward_euler_picard"
    out = []
    for short in (False, True):
        sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
        sim.advance(2)
        if short:
            fill = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
            with pytest.raises(WorldError, match="out of memory"):
                sim.set_neighbor_skin(0.5e-3)
            sim.advance(2)
            del fill
            torch.cuda.empty_cache()
        else:
            sim.advance(2)
        sim.set_neighbor_skin(0.5e-3)
        sim.advance(4)
        out.append((sim.get_state(), sim.get_rhs()))
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("left", [3 << 20, 5 << 20])
def test_asynchronous_copies_survive_a_failed_allocation(left):
    sc = column_collapse(1 << 16, diameters="uniform", mu=0.5, cic=16)
    sc.cfg.neighbor_skin = 0.5e-3              # lists that do not give way
    sc.cfg.kernel_timing = False
    sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
    host = torch.from_numpy(sc.state.copy()).pin_memory()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    with pytest.raises(WorldError, match="out of memory"):
        check(lib.wd_set_state_async(sim.handle, ptr(host)))
    del fill
    torch.cuda.empty_cache()
    sim.advance(2)
    check(lib.wd_set_state_async(sim.handle, ptr(host)))
    sim.synchronize()
    np.testing.assert_array_equal(sim.get_state(), sc.state.reshape(sim.get_state().shape))
    sim.close()


@pytest.mark.parametrize("first", [1, 200])
def test_the_librarys_own_lists_give_way(first):
    """2^18 grains without springs: a checkpoint takes 10 MB, a deposit's accumulators 64, the
    lists that the handle holds for itself 65. Four megabytes are left."""
    n = 1 << 18
    sc = column_collapse(n, diameters="uniform", mu=0.0, cic=64)
    sc.cfg.history = False
    sc.cfg.kernel_timing = False
    out = []
    for short in (False, True):
        sim = ParticleDynamics(sc.cfg, state=sc.state, radius=sc.radius)
        sim.advance(first)
        sim.advance(first)
        fill = short and torch.empty(torch.cuda.mem_get_info()[0] - (4 << 20), dtype=torch.uint8, device="cuda")
        sim.adjoint_record(4, 2)
        sim.advance(40)
        if short:
            assert sim.kernels_per_step() == 6
        del fill
        torch.cuda.empty_cache()
        sim.advance(10)
        sim.set_neighbor_skin(0.5e-3)
        sim.advance(10)
        out.append((sim.get_state(), sim.get_rhs(), sim.compute_momentum(), sim.grid_overflow_count()))
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
