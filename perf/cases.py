"""The workloads this framework is timed on, each through its public entry points.

A case is a dict of plain values. Its "kind" says which calls make up one pass:

  frame     the interactive loop: push a host state, take_step() as often as a rendered
            frame does (drivers.steps_per_frame = 10), unpack_state() to the host
  rollout   upload a state that is on the GPU, advance(steps), read the state back on the
            GPU: restarts, data generation, a surrogate's or controller's inner loop.
            `fields` adds what the data sets store: the CIC density grid and the energy
  batch     the same for many independent scenes of uneven size in one SceneBatch
  fields    the diagnostics of one state without a step: CIC grid, energy, momentum
  gradient  a differentiable window: forward, CIC grid, loss, backward

Scenes ("fill"): `column`, a jittered lattice falling from rest inside a walled box (the
collapse's beginning, hardly any contacts); `packed`, a body-centred lattice whose grains
fly at about half a metre per second with gaps of a percent of their diameter and more, so that
each is soon in contact with one or more neighbours (springs, walls and friction at work).
`skin` 0 searches the grid every step (the default of every configuration file), above 0
it is the Verlet skin in mean diameters. prepare() returns what a program holds before the
call: the handle and the state to start from.

exact() restates the step in float64 torch, from the same inputs, without the library.
"""
from __future__ import annotations

import math

import numpy as np
import torch

D = 5e-3          # mean diameter (m)
DENSITY = 2500.0
GRAVITY = 9.81
K_N = 1e5
CLAMP = K_N * 0.5 * D
DT = 1e-5
CUBE_R = 0.01     # radius, mass and clamp of the default cube scene
CUBE_M = 0.04
CUBE_F = 100.0


def listed():
    return [
        # the default configuration's cube, stepped and shown frame by frame
        {"name": "frame_cube_1k", "kind": "frame", "side": 10, "steps": 10},
        # a small scene rolled out many times: a controller or a design loop
        {"name": "rollout_5k_viscous", "kind": "rollout", "fill": "packed", "n": 5003,
         "diameters": "uniform", "history": False, "mu": 0.5, "skin": 0.1, "steps": 50,
         "picard": 0, "fields": False},
        # the 32,768-grain collapse with a stored field every 100 steps, as configured
        # without any skin
        {"name": "column_32k_stored", "kind": "rollout", "fill": "column", "n": 32768,
         "diameters": "uniform", "history": True, "mu": 0.5, "skin": 0.0, "steps": 100,
         "picard": 0, "fields": True},
        # mid-sized packing, searched every step, odd count
        {"name": "packed_100k_searched", "kind": "rollout", "fill": "packed", "n": 100003,
         "diameters": "uniform", "history": True, "mu": 0.5, "skin": 0.0, "steps": 40,
         "picard": 0, "fields": False},
        # the 2^20-grain collapse from rest, with lists and searched every step
        {"name": "column_1m_lists", "kind": "rollout", "fill": "column", "n": 1 << 20,
         "diameters": "lognormal", "history": True, "mu": 0.5, "skin": 0.15, "steps": 50,
         "picard": 0, "fields": False},
        {"name": "column_1m_searched", "kind": "rollout", "fill": "column", "n": 1 << 20,
         "diameters": "lognormal", "history": True, "mu": 0.5, "skin": 0.0, "steps": 20,
         "picard": 0, "fields": False},
        # a million grains in contact
        {"name": "packed_1m_lists", "kind": "rollout", "fill": "packed", "n": 1000003,
         "diameters": "uniform", "history": True, "mu": 0.5, "skin": 0.15, "steps": 40,
         "picard": 0, "fields": False},
        # the largest: a dense box of equal grains (the 2^24-grain box at a quarter)
        {"name": "packed_4m_lists", "kind": "rollout", "fill": "packed", "n": 1 << 22,
         "diameters": "mono", "history": True, "mu": 0.5, "skin": 0.15, "steps": 20,
         "picard": 0, "fields": False},
        # the implicit integrator on lists, up to 8 iterations
        {"name": "picard_200k", "kind": "rollout", "fill": "packed", "n": 200003,
         "diameters": "uniform", "history": True, "mu": 0.5, "skin": 0.15, "steps": 10,
         "picard": 8, "fields": False},
        # a data-set sweep: uneven scenes stepped together, energies per scene
        {"name": "batch_24_scenes", "kind": "batch", "scenes": 24, "n_min": 4096,
         "n_max": 65536, "history": True, "skin": 0.15, "steps": 40},
        # diagnostics of a large state
        {"name": "fields_1m", "kind": "fields", "n": 1000003, "diameters": "uniform",
         "history": True, "cic": 128},
        # the differentiable window (a shorter one of the 200-step window, same spacing of
        # checkpoints)
        {"name": "gradient_32k", "kind": "gradient", "n": 32768, "steps": 40, "every": 20},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "rollout", "rollout", "rollout", "rollout", "batch", "fields",
                       "gradient"])
    if kind == "frame":
        return {"kind": kind, "side": rng.randint(6, 24), "steps": rng.choice([1, 5, 10, 20])}
    if kind == "batch":
        lo = log_int(1500, 12000)
        return {"kind": kind, "scenes": rng.randint(2, 40), "n_min": lo, "n_max": lo * 8,
                "history": rng.random() < 0.7, "skin": rng.choice([0.0, 0.1, 0.15, 0.2]),
                "steps": rng.randint(8, 40)}
    if kind == "fields":
        return {"kind": kind, "n": log_int(3000, 2500000), "diameters": rng.choice(["mono", "uniform"]),
                "history": rng.random() < 0.7, "cic": rng.choice([32, 63, 64, 100, 128])}
    if kind == "gradient":
        return {"kind": kind, "n": log_int(2000, 60000), "steps": rng.randint(8, 40),
                "every": rng.choice([5, 10, 20])}
    n = log_int(1200, 3000000)
    picard = rng.choice([0, 0, 0, 0, 4, 8])
    most = 30_000_000 // (n * (1 + picard))
    fill = rng.choice(["column", "packed", "packed"])
    return {"kind": kind, "fill": fill, "n": n,
            "diameters": rng.choice(["mono", "uniform"] if fill == "packed" else ["uniform", "lognormal"]),
            "history": rng.random() < 0.7, "mu": round(rng.uniform(0.1, 0.8), 3),
            "skin": rng.choice([0.0, 0.0, 0.1, 0.15, 0.2]),
            "steps": max(3, min(most, rng.randint(10, 100))), "picard": picard,
            "fields": rng.random() < 0.25}


# ---- scenes --------------------------------------------------------------------------

class Scene:
    """State [n, 6] and radii (float32, host) with the physics of one box."""

    def __init__(self, state, radius, mass, lo, hi, grid, mu, history):
        self.state, self.radius, self.mass = state, radius, mass
        self.lo, self.hi, self.grid = lo, hi, grid
        self.mu, self.history = mu, history and mu > 0
        self.k_n, self.f_max, self.dt, self.e = K_N, CLAMP, DT, 0.5
        self.picard, self.picard_tol, self.cic = 0, 0.0, (32, 32, 32)


def _diameters(rng, n, kind):
    if kind == "mono":
        return np.full(n, D)
    if kind == "uniform":
        return rng.uniform(0.9 * D, 1.1 * D, n)
    return np.clip(rng.lognormal(math.log(D) - 0.5 * 0.15 ** 2, 0.15, n), 0.7 * D, 1.4 * D)


def _sphere_mass(radius):
    r = radius.astype(np.float64)
    return (DENSITY * 4.0 / 3.0 * np.pi * r * r * r).astype(np.float32)


def _finish(pos, vel, diam, box, mu, history):
    state = np.concatenate([pos, vel], axis=1).astype(np.float32)
    radius = (0.5 * diam).astype(np.float32)
    lo = np.array([-0.5 * box[0], -0.5 * box[1], 0.0], np.float32)
    hi = np.array([0.5 * box[0], 0.5 * box[1], box[2]], np.float32)
    cell = max(1.1 * D, float(diam.max()))
    grid = [max(1, int(b // cell)) for b in box]
    return Scene(state, radius, _sphere_mass(radius), lo, hi, grid, mu, history)


def column(n, kind, mu, history, seed):
    """n sites of a simple cubic lattice in a cylinder of height 4R, jittered, at rest."""
    rng = np.random.default_rng(seed)
    scale = (n / 32768.0) ** (1.0 / 3.0)
    radius, box = 0.1 * scale, (1.0 * scale, 1.0 * scale, 0.5 * scale)
    diam = _diameters(rng, n, kind)
    dmax = float(diam.max())
    step = max((math.pi * radius * radius * 4 * radius / n) ** (1.0 / 3.0), 1.001 * dmax)
    ax = np.arange(-math.ceil(radius / step), math.ceil(radius / step) + 1) * step
    yy, xx = np.meshgrid(ax, ax, indexing="ij")
    inside = xx * xx + yy * yy <= radius * radius
    layer = np.stack([xx[inside], yy[inside]], axis=1)
    layers = -(-n // len(layer))
    z = 0.5 * (step + dmax) + step * np.arange(layers)
    box = (box[0], box[1], max(box[2], float(z[-1]) + dmax))
    pos = np.concatenate([np.tile(layer, (layers, 1)), np.repeat(z, len(layer))[:, None]], axis=1)[:n]
    pos = pos + rng.uniform(-0.05 * D, 0.05 * D, (n, 3))
    return _finish(pos, np.zeros((n, 3)), diam, box, mu, history)


def packed(n, kind, mu, history, seed):
    """n sites of a body-centred lattice filling a box, jittered, flying at N(0, 0.5 m/s)."""
    rng = np.random.default_rng(seed)
    diam = _diameters(rng, n, kind)
    a = 2.0 / math.sqrt(3.0) * 1.01 * (float(diam.max()) + D) / 2
    m = math.ceil((n / 2) ** (1.0 / 3.0))
    i = np.arange(n, dtype=np.int64)
    c, half = i // 2, (i % 2)[:, None]
    pos = np.stack([c % m, c // m % m, c // (m * m)], axis=1) * a + half * (0.5 * a)
    pos = pos + rng.uniform(-0.01 * D, 0.01 * D, (n, 3)) + 0.52 * float(diam.max())
    side = (m - 0.5) * a + 1.05 * float(diam.max())
    box = (side, side, 1.25 * side)
    pos[:, :2] -= 0.5 * side
    return _finish(pos, rng.normal(0.0, 0.5, (n, 3)), diam, box, mu, history)


def cube(side, seed):
    """The default scene: side^3 grains of the default radius and mass, jittered."""
    rng = np.random.default_rng(seed)
    n = side ** 3
    i = np.arange(n)
    pos = np.stack([i // (side * side), i // side % side, i % side], axis=1) * (2 * CUBE_R)
    pos = pos - CUBE_R * (side - 1) + rng.uniform(-0.3 * CUBE_R, 0.3 * CUBE_R, (n, 3))
    s = Scene(np.concatenate([pos, np.zeros((n, 3))], axis=1).astype(np.float32),
              np.full(n, CUBE_R, np.float32), np.full(n, CUBE_M, np.float32),
              np.full(3, -1.0, np.float32), np.full(3, 1.0, np.float32), [32] * 3, 0.5, False)
    s.k_n, s.f_max, s.dt, s.e = CUBE_F / float(np.float32(CUBE_R)), CUBE_F, 1e-4, 0.3
    return s


def scenes_of(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return [cube(case["side"], seed)]
    if kind == "batch":
        rng = np.random.default_rng([seed, 1])
        ns = np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["scenes"]))
        # the counts are the case's, not the seed's: every seed has the same work
        ns = case["n_min"] * (case["n_max"] / case["n_min"]) ** ((np.argsort(np.argsort(ns)) + 0.5) / len(ns))
        mus = rng.uniform(0.1, 0.8, case["scenes"])
        return [(packed if k % 2 else column)(int(ns[k]), "uniform", float(mus[k]),
                                              case["history"], [seed, 2, k])
                for k in range(case["scenes"])]
    if kind == "fields":
        s = packed(case["n"], case["diameters"], 0.5, case["history"], seed)
        s.cic = (case["cic"],) * 3
    elif kind == "gradient":
        s = packed(case["n"], "uniform", 0.5, True, seed)
        s.cic = (64, 64, 64)
    else:
        make = column if case["fill"] == "column" else packed
        s = make(case["n"], case["diameters"], case["mu"], case["history"], seed)
        s.cic = (64, 64, 64)
        s.picard, s.picard_tol = case["picard"], 1e-6 if case["picard"] else 0.0
    return [s]


# ---- through the library --------------------------------------------------------------

def _config(s, skin):
    from world_b200 import SimConfig
    cfg = SimConfig()
    ph = cfg.physics
    for a, ax in enumerate("xyz"):
        setattr(cfg.domain, ax + "_min", float(s.lo[a]))
        setattr(cfg.domain, ax + "_max", float(s.hi[a]))
        setattr(cfg, "collision_grid_size_" + ax, s.grid[a])
        setattr(cfg, "density_grid_size_" + ax, s.cic[a])
    ph.wall_x_min, ph.wall_y_min, ph.floor_z = (float(v) for v in s.lo)
    ph.wall_x_max, ph.wall_y_max, ph.ceiling_z = (float(v) for v in s.hi)
    ph.gravity, ph.particle_radius = GRAVITY, 0.5 * D
    ph.normal_stiffness, ph.max_force = s.k_n, s.f_max
    ph.restitution, ph.friction, ph.density = s.e, s.mu, DENSITY
    cfg.history, cfg.dt, cfg.particles_per_cell = s.history, s.dt, 16
    cfg.neighbor_skin, cfg.kernel_timing = skin * D, False
    if s.picard:
        cfg.time_integrator = "backward_euler_picard"
        cfg.picard_iterations, cfg.picard_tolerance = s.picard, s.picard_tol
    return cfg


def prepare(case, seed):
    from world_b200 import ParticleDynamics, SceneBatch, SimConfig
    kind, scenes = case["kind"], scenes_of(case, seed)
    s = scenes[0]
    st = {"case": case}
    if kind == "frame":
        # every setting at its default, kernel timing included
        st["sim"] = ParticleDynamics(SimConfig(), state=s.state)
        st["start"] = s.state.reshape(-1)
        return st
    skin = case.get("skin", 0.0)
    if kind == "batch":
        st["sim"] = SceneBatch([_config(x, skin) for x in scenes], [x.state for x in scenes],
                               radii=[x.radius for x in scenes])
    else:
        st["sim"] = ParticleDynamics(_config(s, skin), state=s.state, radius=s.radius)
    st["start"] = torch.from_numpy(np.concatenate([x.state.reshape(-1) for x in scenes])).cuda()
    st["out"] = torch.empty_like(st["start"])
    if kind == "fields":
        st["grid"] = torch.empty(4 * case["cic"] ** 3, dtype=torch.float32, device="cuda")
    if kind == "gradient":
        x = st["start"].reshape(-1, 6)
        st["x0"], st["v0"] = x[:, :3].contiguous(), x[:, 3:].contiguous()
        st["theta"] = torch.tensor([0.5, 0.5, K_N], dtype=torch.float32)
        target = np.random.default_rng([seed, 3]).uniform(0.5, 1.5, s.cic)
        st["target"] = torch.from_numpy(target.astype(np.float32)).cuda() * _mean_mass(s)
    return st


def _mean_mass(s):
    return float(s.mass.sum() / np.prod(s.cic))


def run(st):
    case, sim = st["case"], st["sim"]
    kind = case["kind"]
    if kind == "frame":
        sim.device_state.copy_from_host(st["start"])
        for _ in range(case["steps"]):
            sim.take_step()
        sim.unpack_state()
        return sim.host_state
    if kind == "fields":
        from world_b200._lib import check, lib, ptr
        check(lib.wd_compute_density_grid_device(sim.handle, ptr(st["grid"])))
        return {"grid": st["grid"], "energy": sim.compute_total_energy(),
                "momentum": sim.compute_momentum()}
    if kind == "gradient":
        from world_b200.adjoint import deposit, window
        x0 = st["x0"].detach().requires_grad_(True)
        v0 = st["v0"].detach().requires_grad_(True)
        theta = st["theta"].detach().requires_grad_(True)
        x, v = window(sim, x0, v0, theta, steps=case["steps"], checkpoint_every=case["every"])
        grid = deposit(sim, x, v)
        loss = ((grid[0] - st["target"]) ** 2).sum()
        loss.backward()
        return {"x": x.detach(), "v": v.detach(), "grid": grid.detach(), "gx": x0.grad,
                "gv": v0.grad, "gtheta": theta.grad}
    sim.set_state_tensor(st["start"])
    sim.advance(case["steps"])
    out = {"state": sim.state_tensor(st["out"])}
    if kind == "batch":
        out["energies"] = sim.scene_energies()
    elif case["fields"]:
        sim.compute_density_grid()
        out["grid"] = sim.host_density_grid
        out["energy"] = sim.compute_total_energy()
    return out


def _counts(case):
    if case["kind"] == "frame":
        return case["side"] ** 3
    if case["kind"] == "batch":
        r = case["n_max"] / case["n_min"]
        k = case["scenes"]
        return sum(int(case["n_min"] * r ** ((i + 0.5) / k)) for i in range(k))
    return case["n"]


def work(case):
    """Per step and grain: position, radius, velocity and mass read, position and velocity
    written (56 bytes), gravity, walls, integration and a handful of neighbours. A window's
    backward reads each step's state again and carries adjoints of the same size."""
    n, kind = _counts(case), case["kind"]
    if kind == "fields":
        nodes = case["cic"] ** 3
        return {"bytes": 3 * 32 * n + 16 * nodes, "flops": 250 * n}
    steps = case["steps"] * max(1, case.get("picard", 0) // 2)
    per = 56 * (3 if kind == "gradient" else 1)
    extra = 16 * 64 ** 3 if case.get("fields") or kind == "gradient" else 0
    return {"bytes": n * (steps * per + 48) + extra, "flops": n * steps * 250 * (4 if kind == "gradient" else 1)}


# ---- the same in float64 --------------------------------------------------------------

class _Exact:
    """One scene stepped in float64 (torch): pairs kept within a margin, springs per pair."""

    MARGIN = 0.2

    def __init__(self, s):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def up(a):
            return torch.from_numpy(np.asarray(a)).to(dev, torch.float64)

        f = lambda v: float(np.float32(v))  # noqa: E731  the library's inputs are float32
        self.dev, self.s = dev, s
        self.x, self.v = up(s.state[:, :3]), up(s.state[:, 3:])
        self.r, self.m = up(s.radius), up(s.mass)
        self.lo, self.hi = up(s.lo), up(s.hi)
        self.dt, self.g, self.f_max = f(s.dt), f(GRAVITY), f(s.f_max)
        self.mu = torch.tensor(f(s.mu), dtype=torch.float64, device=dev)
        self.e = torch.tensor(f(s.e), dtype=torch.float64, device=dev)
        self.k = torch.tensor(f(s.k_n), dtype=torch.float64, device=dev)
        self.wall_xi = torch.zeros(6, self.x.shape[0], 3, dtype=torch.float64, device=dev)
        self.pairs = None

    def near(self):
        """Pairs closer than their radii plus the margin; springs follow their pairs."""
        x = self.x.detach()
        margin = self.MARGIN * 2 * float(self.r.mean())
        if self.pairs is not None and float((x - self.built).norm(dim=1).max()) < 0.49 * margin:
            return
        n = x.shape[0]
        w = 2 * float(self.r.max()) + margin
        c = ((x - x.min(0).values) / w).long() + 1
        dims = (c.max(0).values + 2).tolist()
        key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
        key, order = key.sort()
        cells, count = torch.unique_consecutive(key, return_counts=True)
        first = count.cumsum(0) - count
        most, slot = int(count.max()), torch.arange(n, device=self.dev)
        found = []
        for dx in (0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    off = (dx * dims[1] + dy) * dims[2] + dz
                    if off < 0:
                        continue
                    at = torch.searchsorted(cells, key + off).clamp_(max=cells.numel() - 1)
                    hit = cells[at] == key + off
                    for q in range(most):
                        j = first[at] + q
                        ok = (hit & (q < count[at]) & ((j > slot) if off == 0 else hit)).nonzero()[:, 0]
                        a, b = order[ok], order[j[ok]]
                        a, b = torch.minimum(a, b), torch.maximum(a, b)
                        near = (x[a] - x[b]).square().sum(1) < (self.r[a] + self.r[b] + margin).square()
                        found.append(a[near] * n + b[near])
        code = torch.cat(found).sort().values
        xi = torch.zeros(code.numel(), 3, dtype=torch.float64, device=self.dev)
        if self.pairs is not None and self.code.numel():
            at = torch.searchsorted(code, self.code).clamp_(max=max(0, code.numel() - 1))
            same = code[at] == self.code
            xi[at[same]] = self.xi[same]
        self.code, self.pairs, self.xi, self.built = code, (code // n, code % n), xi, x.clone()

    def damping(self, mass):
        ln = torch.log(self.e)
        return -2 * torch.sqrt(mass * self.k) * ln / torch.sqrt(math.pi ** 2 + ln * ln)

    def friction(self, vt, nrm, limit, c, xi):
        """(force, new spring) of the tangential law."""
        if not self.s.history:
            v = vt.square().sum(1).sqrt()
            mag = torch.minimum(limit, c * v)
            slow = v < 1e-8
            return torch.where(slow[:, None], torch.zeros_like(vt),
                               -mag[:, None] * vt / torch.where(slow, torch.ones_like(v), v)[:, None]), xi
        xi = xi - (xi * nrm).sum(1, keepdim=True) * nrm + self.dt * vt
        ft = -(2.0 / 7.0) * self.k * xi
        f2 = ft.square().sum(1)
        slip = f2 > limit * limit
        scale = torch.where(slip, limit / torch.where(slip, f2, torch.ones_like(f2)).sqrt(), torch.ones_like(f2))
        return ft * scale[:, None], xi * scale[:, None]

    def forces(self, x, v):
        """(force, pair springs, wall springs) at (x, v) from the stored springs."""
        f = torch.zeros_like(x)
        f = f + torch.stack([torch.zeros_like(self.m), torch.zeros_like(self.m), -self.m * self.g], 1)
        wall = torch.zeros_like(self.wall_xi)
        for a in range(3):
            for up in (0, 1):
                d = (self.hi[a] - x[:, a] if up else x[:, a] - self.lo[a]) - self.r
                t = (d < 0).nonzero()[:, 0]
                if not t.numel():
                    continue
                nrm = torch.zeros(t.numel(), 3, dtype=torch.float64, device=self.dev)
                nrm[:, a] = -1.0 if up else 1.0
                fn = (-self.k * d[t]).clamp(0, self.f_max)
                c = self.damping(self.m[t])
                vn = v[t, a:a + 1]
                axis = nrm.abs()
                vt = v[t] - vn * axis
                ft, xi = self.friction(vt, nrm, self.mu * fn, c, self.wall_xi[2 * a + up][t])
                f = f.index_add(0, t, fn[:, None] * nrm - c[:, None] * vn * axis + ft)
                wall[2 * a + up, t] = xi.detach() if not xi.requires_grad else xi
        i, j = self.pairs
        with torch.no_grad():
            touch = ((x[i] - x[j]).square().sum(1) < (self.r[i] + self.r[j]).square()).nonzero()[:, 0]
        i, j = i[touch], j[touch]
        d = x[i] - x[j]
        norm = d.square().sum(1).sqrt()
        nrm = d / norm[:, None]
        fn = (self.k * (self.r[i] + self.r[j] - norm)).clamp(0, self.f_max)
        c = self.damping(self.m[i] * self.m[j] / (self.m[i] + self.m[j]))
        vr = v[i] - v[j]
        vn = (vr * nrm).sum(1, keepdim=True)
        ft, xi = self.friction(vr - vn * nrm, nrm, self.mu * fn, c, self.xi[touch])
        p = fn[:, None] * nrm - c[:, None] * vn * nrm + ft
        f = f.index_add(0, i, p).index_add(0, j, -p)
        springs = torch.zeros_like(self.xi).index_add(0, touch, xi)
        return f, springs, wall

    def step(self):
        self.near()
        if not self.s.picard:
            f, self.xi, self.wall_xi = self.forces(self.x, self.v)
            self.v = self.v + self.dt * f / self.m[:, None]
            self.x = self.x + self.dt * self.v
            return
        x, v = self.x, self.v
        for _ in range(self.s.picard):
            f, xi, wall = self.forces(x, v)
            v = self.v + self.dt * f / self.m[:, None]
            last, x = x, self.x + self.dt * v
            if float((x - last).abs().max()) < self.s.picard_tol:
                break
        self.x, self.v, self.xi, self.wall_xi = x, v, xi, wall

    def state(self):
        return torch.cat([self.x, self.v], dim=1).reshape(-1)

    def energy(self):
        self.near()
        cd = self.f_max / float(self.k)

        def spring(d):
            d = d.clamp(min=0)
            inner = 0.5 * self.k * d * d
            return torch.where(d <= cd, inner, 0.5 * self.f_max * cd + self.f_max * (d - cd)).sum()

        e = (0.5 * self.m * self.v.square().sum(1)).sum()
        e = e + (self.m * self.g * (self.x[:, 2] - self.lo[2])).sum()
        for a in range(3):
            e = e + spring(self.r - (self.x[:, a] - self.lo[a])) + spring(self.r - (self.hi[a] - self.x[:, a]))
        i, j = self.pairs
        e = e + spring(self.r[i] + self.r[j] - (self.x[i] - self.x[j]).square().sum(1).sqrt())
        if self.s.history:
            e = e + 0.5 * (2.0 / 7.0) * self.k * (self.xi.square().sum() + self.wall_xi.square().sum())
        return e

    def grid(self):
        size = torch.tensor(self.s.cic, device=self.dev)
        u = (self.x - self.lo) / ((self.hi - self.lo) / (size - 1))
        base = u.detach().floor()
        w = u - base
        q = torch.cat([self.m[:, None], self.m[:, None] * self.v], dim=1)
        out = torch.zeros(int(np.prod(self.s.cic)), 4, dtype=torch.float64, device=self.dev)
        for corner in range(8):
            b = torch.tensor([corner >> 2 & 1, corner >> 1 & 1, corner & 1], device=self.dev)
            k = torch.minimum((base.long() + b).clamp(min=0), size - 1)
            node = (k[:, 0] * size[1] + k[:, 1]) * size[2] + k[:, 2]
            out = out.index_add(0, node, q * torch.where(b > 0, w, 1 - w).prod(1)[:, None])
        return out.t().contiguous()


def exact(case, seed):
    kind, scenes = case["kind"], scenes_of(case, seed)
    sims = [_Exact(s) for s in scenes]
    e = sims[0]
    if kind == "fields":
        return {"grid": e.grid().reshape(-1), "energy": float(e.energy()),
                "momentum": (e.m[:, None] * e.v).sum(0)}
    if kind == "gradient":
        s = scenes[0]
        e.x, e.v = e.x.requires_grad_(True), e.v.requires_grad_(True)
        x0, v0 = e.x, e.v
        theta = [t.requires_grad_(True) for t in (e.mu, e.e, e.k)]
        target = np.random.default_rng([seed, 3]).uniform(0.5, 1.5, s.cic).astype(np.float32)
        target = torch.from_numpy(target).to(e.dev) * torch.tensor(_mean_mass(s), dtype=torch.float32)
        for _ in range(case["steps"]):
            e.step()
        grid = e.grid().reshape(4, *s.cic)
        ((grid[0] - target.double()) ** 2).sum().backward()
        return {"x": e.x.detach(), "v": e.v.detach(), "grid": grid.detach(), "gx": x0.grad, "gv": v0.grad,
                "gtheta": torch.stack([t.grad for t in theta])}
    for x in sims:
        for _ in range(case["steps"]):
            x.step()
    state = torch.cat([x.state() for x in sims])
    if kind == "frame":
        return state
    if kind == "batch":
        return {"state": state, "energies": torch.stack([x.energy() for x in sims])}
    if case["fields"]:
        return {"state": state, "grid": e.grid().reshape(-1), "energy": float(e.energy())}
    return {"state": state}
