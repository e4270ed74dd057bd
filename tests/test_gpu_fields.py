"""The CIC deposit's kernel at the edges of its groups (32 lanes, 128 grains a warp, 512 a
block), with grains outside the box, massless and negative masses, and channel scales whose
power of two is no float: against float64 sums of the same float32 products. Each node is
the correctly rounded sum up to 2^-62 of the channel's bound per contribution, so it differs
from the float64 sum by half an ulp of float32 and that quantum."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import packed_poly
from world_b200 import ParticleDynamics

pytestmark = pytest.mark.gpu


def _field(st, m, lo, hi, size):
    f32 = np.float32
    out = np.zeros((4, size ** 3))
    h = [f32((f32(hi) - f32(lo)) / f32(size - 1))] * 3
    u = [((st[:, a] - f32(lo)) / h[a]).astype(f32) for a in range(3)]
    base = [np.floor(x) for x in u]
    w = [(f32(1) - (x - b).astype(f32), (x - b).astype(f32)) for x, b in zip(u, base)]
    part = [m] + [(m * st[:, 3 + a]).astype(f32) for a in range(3)]
    for c in range(8):
        k = [(c >> 2) & 1, (c >> 1) & 1, c & 1]
        i = [np.clip(base[a] + k[a], 0, size - 1).astype(np.int64) for a in range(3)]
        wt = ((w[0][k[0]] * w[1][k[1]]).astype(f32) * w[2][k[2]]).astype(f32)
        for q in range(4):
            np.add.at(out[q], (i[0] * size + i[1]) * size + i[2], (part[q] * wt).astype(f32).astype(np.float64))
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 511, 513, 2500])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e30])
def test_deposit_is_the_rounded_sum(n, scale):
    cfg, st, rad = packed_poly(n=n, seed=70)
    st = st.astype(np.float32)
    if n > 100:
        st[:7, 0] = -0.07                       # outside the box: clamped to its edge nodes
        st[7:14, 2] = 0.09
    rng = np.random.default_rng(71)
    m = (rng.uniform(0.5, 1.5, n) * scale).astype(np.float32)
    m[n // 2:n // 2 + 3] = 0.0
    m[-1] = -m[-1]
    sim = ParticleDynamics(cfg, state=st, radius=rad, mass=m)
    sim.compute_density_grid()
    got = sim.host_density_grid.reshape(4, -1).astype(np.float64)
    size = cfg.density_grid_size_x
    want = _field(st, m, cfg.domain.x_min, cfg.domain.x_max, size)
    for c in range(4):
        bound = n * np.abs(m if c == 0 else m * st[:, 2 + c]).max()
        tol = 2.0 ** -24 * np.abs(want[c]) + n * 2.0 ** -52 * bound
        assert (np.abs(got[c] - want[c]) <= tol).all(), c
    first = sim.host_density_grid.copy()
    sim.compute_density_grid()
    np.testing.assert_array_equal(first, sim.host_density_grid)
    e = [sim.compute_total_energy() for _ in range(3)]   # direct, then as device graphs
    assert e[0] == e[1] == e[2] == pytest.approx(sim.grain_energies().sum(), rel=1e-12)
    sim.close()


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 33, 257])
def test_states_on_any_float_alignment(n, offset):
    """States in and out of CUDA tensors that start on 4, 8 or 16 bytes, after a step has
    re-ordered the slots: copies, so equal to the bit, with nothing written beside them."""
    import torch
    cfg, st, rad = packed_poly(n=n, seed=68)
    sim = ParticleDynamics(cfg, state=st, radius=rad)
    sim.advance(1)
    want = np.random.default_rng(69).uniform(-0.01, 0.01, 6 * n).astype(np.float32)
    buf = torch.zeros(6 * n + 8, device="cuda")
    buf[offset:offset + 6 * n] = torch.from_numpy(want).cuda()
    sim.set_state_tensor(buf[offset:offset + 6 * n])
    out = torch.full((6 * n + 8,), 7.0, device="cuda")
    sim.state_tensor(out[offset:offset + 6 * n])
    got = out.cpu().numpy()
    assert np.array_equal(got[offset:offset + 6 * n], want)
    assert np.all(got[:offset] == 7.0) and np.all(got[offset + 6 * n:] == 7.0)
