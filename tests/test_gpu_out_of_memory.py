"""A call that finds too little device memory returns an error, once, and leaves the library
usable."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from world_b200 import ParticleDynamics, WorldError
from world_b200.scenes import column_collapse

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once():
    sc = column_collapse(1 << 16, diameters="uniform", mu=0.5, cic=16)
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
