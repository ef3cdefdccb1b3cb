"""The work whose speed this repository watches: calls through the public
entry points, over the sizes, options and directions that they are used in.

- ``sph``: one ``SolverSPH.step``, from a few thousand particles (where the
  launches count) to the 128^3 block; with the density and pressure outputs,
  an external force, inactive particles and the tolerance arithmetic.
- ``worlds``: one step of many independent scenes in one solver.
- ``rollout``: a checkpointed differentiable rollout, forward and backward.
- ``surrogate``: one call of the learned large-step surrogate.
- ``contact``: the penalty-contact particle step (grid build, particle
  contacts, integration).
- ``xpbd``: the position-based particle step with a ground plane.
- ``raycast``: a depth image of a particle block.
- ``hashgrid``: a grid build and a batched query.

Fluid inputs are blocks of particles near rest density, disordered and warped
so that the lattice is not aligned with the grid's cells, as a running
simulation leaves them, in the index order in which a scene is built.
"""

from __future__ import annotations

import math
import os

import numpy as np
import torch

DEV = "cuda:0" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # a desk-top scene or one environment of a controller: launches and latency
        dict(name="step_2k", kind="sph", nx=13, ny=12, nz=13, s=0.02, bx=0.6, by=0.4, bz=0.6, dt=2e-4),
        # the 32^3 dam break, recording density and pressure
        dict(name="step_32k", kind="sph", nx=32, ny=32, nz=32, s=0.01, bx=1.0, by=1.0, bz=1.0, dt=1e-4, fields=True),
        # a ragged block with an external force and some inactive particles, tolerance arithmetic
        dict(name="step_219k_fast", kind="sph", nx=97, ny=61, nz=37, s=0.007, bx=1.5, by=0.6, bz=0.8, dt=7e-5,
             force=True, inactive=0.02, fast=True),
        # the 1M tank of the benchmark
        dict(name="step_1m", kind="sph", nx=128, ny=128, nz=64, s=0.005, bx=2.0, by=1.0, bz=1.0, dt=5e-5),
        # the 128^3 block in the same tank
        dict(name="step_2m", kind="sph", nx=128, ny=128, nz=128, s=0.005, bx=2.0, by=1.0, bz=1.0, dt=5e-5),
        # batched scenes of 256 to 16384 particles, each with its own spacing
        dict(name="worlds_512", kind="worlds", worlds=512, dt=1e-4),
        # gradients of a rollout with respect to the initial state and the stiffness
        dict(name="rollout_grad_64k", kind="rollout", nx=64, ny=64, nz=16, s=0.01, bx=1.0, by=1.0, bz=1.0, dt=1e-4,
             steps=20, every=10),
        # the learned step of 4 x dt on a 64^3 block
        dict(name="surrogate_262k", kind="surrogate", nx=64, ny=64, nz=64, s=0.005, bx=0.8, by=0.5, bz=0.8, dt=5e-5),
        # 1M touching spheres: grid build, particle contacts, integration
        dict(name="contact_1m", kind="contact", nx=128, ny=128, nz=64, s=0.0095, r=0.005, dt=1e-4),
        # a pile on the ground, position-based, 4 iterations
        dict(name="xpbd_262k", kind="xpbd", nx=64, ny=64, nz=64, s=0.0095, r=0.005, dt=1e-3, iters=4),
        # a 640 x 480 depth image of half a million spheres
        dict(name="raycast_640x480", kind="raycast", nx=101, ny=100, nz=51, s=0.0095, r=0.005, width=640, height=480),
        # a grid over scattered points and a query of some of them
        dict(name="hashgrid_300k", kind="hashgrid", n=300007, q=40001, extent=1.3, radius=0.02, dim=128),
    ]


def _split(rng, n):
    """Three ragged dimensions whose product is near n."""
    a = max(3, round((n ** (1 / 3)) * rng.uniform(0.7, 1.4)))
    b = max(3, round(math.sqrt(n / a) * rng.uniform(0.7, 1.4)))
    return a, b, max(3, round(n / (a * b)))


def draw(rng):
    kind = rng.choice(["sph", "sph", "sph", "worlds", "rollout", "surrogate", "contact", "xpbd", "raycast", "hashgrid"])

    def size(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    if kind == "worlds":
        return dict(kind=kind, worlds=round(size(8, 400)), dt=1e-4)
    if kind == "hashgrid":
        n = round(size(1000, 1000000))
        return dict(kind=kind, n=n, q=max(1, n // 8), extent=round(rng.uniform(0.5, 2.5), 3),
                    radius=round(rng.uniform(0.01, 0.03), 4), dim=rng.choice([64, 100, 128]))
    top = {"sph": 1900000, "rollout": 60000, "surrogate": 240000, "contact": 1000000, "xpbd": 250000,
           "raycast": 500000}[kind]
    nx, ny, nz = _split(rng, size(1000, top))
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind in ("contact", "xpbd", "raycast"):
        c.update(s=0.0095, r=0.005, dt=1e-4 if kind == "contact" else 1e-3)
        if kind == "xpbd":
            c.update(iters=rng.choice([1, 2, 3, 4]))
        if kind == "raycast":
            c.update(width=rng.randint(60, 600), height=rng.randint(60, 460))
            del c["dt"]
        return c
    s = round(rng.uniform(0.004, 0.02), 4)
    bx, by, bz = ((k + 3) * s * rng.uniform(1.0, most) for k, most in ((nx, 2.5), (ny, 1.6), (nz, 2.5)))
    c.update(s=s, bx=round(bx, 3), by=round(by, 3), bz=round(bz, 3), dt=0.01 * s)
    if kind == "sph":
        c.update(fields=rng.random() < 0.3, force=rng.random() < 0.3, fast=rng.random() < 0.2,
                 inactive=0.03 if rng.random() < 0.3 else 0.0)
    if kind == "rollout":
        c.update(steps=rng.randint(2, 18), every=rng.choice([1, 4, 10]))
    return c


# ---------------------------------------------------------------------------
# inputs (functions of the case and the seed alone)
# ---------------------------------------------------------------------------
def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _lattice(nx, ny, nz):
    """Indices in the order of a scene's lattice: iy slowest, then ix, then iz."""
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz)), -1).reshape(-1, 3)
    return g.astype(np.float32)


def _fluid(case, seed):
    """Positions, velocities (N, 3) float32, flags, external force or None."""
    rng = _rng(seed)
    s = case["s"]
    x = (_lattice(case["nx"], case["ny"], case["nz"]) + 0.5) * np.float32(s)
    ph = rng.uniform(0, 2 * math.pi, 3)
    warp = np.empty_like(x)
    for a in range(3):
        warp[:, a] = 0.3 * s * np.sin(x[:, (a + 1) % 3] * (2 * math.pi / (13 * s)) + ph[a])
    x += warp
    x += rng.uniform(0, s, 3).astype(np.float32) + np.float32(0.4 * s)
    x += (rng.random(x.shape, dtype=np.float32) - np.float32(0.5)) * np.float32(0.16 * s)
    v = rng.standard_normal(x.shape, dtype=np.float32) * np.float32(0.05)
    n = len(x)
    flags = np.ones(n, dtype=np.int32)
    if case.get("inactive"):
        flags[rng.random(n) < case["inactive"]] = 0
    f = None
    if case.get("force"):
        f = rng.standard_normal(x.shape, dtype=np.float32) * np.float32(5.0 * 1000.0 * s ** 3)
    return x, v, flags, f


def _spheres(case, seed):
    """Touching spheres on a jittered lattice: positions, velocities, radii."""
    rng = _rng(seed, 1)
    s, r = case["s"], case["r"]
    x = (_lattice(case["nx"], case["ny"], case["nz"]) + 0.5) * np.float32(s)
    x[:, :2] += rng.uniform(0, s, 2).astype(np.float32)
    x += (rng.random(x.shape, dtype=np.float32) - np.float32(0.5)) * np.float32(0.2 * s)
    v = rng.standard_normal(x.shape, dtype=np.float32) * np.float32(0.1)
    rad = np.float32(r) * (np.float32(0.9) + np.float32(0.1) * rng.random(len(x), dtype=np.float32))
    return x, v, rad


def _worlds(case, seed):
    """Per world (positions, spacing): 256 to 16384 particles each (the sizes
    and spacings belong to the case, the particles to the seed)."""
    plan, rng = _rng(case["worlds"], 5), _rng(seed, 2)
    out = []
    for n in np.exp(plan.uniform(math.log(256), math.log(16384), case["worlds"])):
        a = max(2, int(n ** (1 / 3)))
        s = float(plan.uniform(0.004, 0.01))
        x = (_lattice(a, a, max(1, round(n / (a * a)))) + 0.5) * np.float32(s)
        x += rng.uniform(0, s, 3).astype(np.float32) + np.float32(0.4 * s)
        x += (rng.random(x.shape, dtype=np.float32) - np.float32(0.5)) * np.float32(0.2 * s)
        out.append((x, s))
    return out


def _scatter(case, seed):
    """Points at random over a cube, in random order; the first q are the
    queries. The number of points in each cell belongs to the case (so that
    the query finds the same total), their places and order to the seed."""
    plan, rng = _rng(case["n"], 6), _rng(seed, 3)
    n, q, r = case["n"], case["q"], case["radius"]
    cell = plan.integers(0, max(1, int(case["extent"] / r)), (n, 3))
    order = np.concatenate([rng.permutation(q), q + rng.permutation(n - q)])
    return ((cell[order] + 0.1 + 0.8 * rng.random((n, 3))) * r).astype(np.float32)


WORLD_BOX = 0.5


def _camera(case):
    """A camera that sees the block obliquely from outside."""
    e = np.array([case["nx"], case["ny"], case["nz"]], dtype=np.float64) * case["s"]
    t = 0.5 * e
    far = 1.7 * float(np.linalg.norm(e)) + 0.2
    d = np.array([0.62, -0.6, 0.5])
    pos = t + d / np.linalg.norm(d) * far
    return pos, t - pos, far * 1.7


# ---------------------------------------------------------------------------
# what a user's program has in hand before the call
# ---------------------------------------------------------------------------
def _config(case):
    from newton_sph_dev_b200.solvers import SolverSPH

    return SolverSPH.Config(smoothing_length=2 * case["s"], rest_density=1000.0, sound_speed=20.0, eos_gamma=7,
                            xsph=0.01, box_lo=(0.0, 0.0, 0.0), box_hi=(case["bx"], case["by"], case["bz"]),
                            arithmetic="fast" if case.get("fast") else "exact")


def prepare(case, seed):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSemiImplicit, SolverSPH, SolverXPBD

    kind = case["kind"]
    b = nsph.ModelBuilder()
    if kind == "hashgrid":
        pts = torch.from_numpy(_scatter(case, seed)).to(DEV)
        qs = pts[:case["q"]].contiguous()
        grid = nsph.HashGrid(case["dim"], case["dim"], case["dim"], device=DEV)
        grid.reserve(case["n"])
        return dict(kind=kind, grid=grid, pts=pts, qs=qs, radius=case["radius"])
    if kind == "worlds":
        cfgs = []
        for x, s in _worlds(case, seed):
            b.begin_world()
            b.add_particles(pos=x, vel=np.zeros_like(x), mass=np.full(len(x), 1000.0 * s ** 3))
            b.end_world()
            cfgs.append(SolverSPH.Config(smoothing_length=2 * s, rest_density=1000.0, sound_speed=20.0, eos_gamma=7,
                                         xsph=0.01, box_lo=(0.0, 0.0, 0.0), box_hi=(WORLD_BOX,) * 3))
        model = b.finalize(DEV)
        return dict(kind="sph", solver=SolverSPH(model, cfgs), s0=model.state(), s1=model.state(), dt=case["dt"])
    if kind in ("contact", "xpbd", "raycast"):
        x, v, rad = _spheres(case, seed)
        b.add_particles(pos=x, vel=v, mass=np.full(len(x), 1.0), radius=rad)
        if kind == "xpbd":
            b.add_ground_plane()
        model = b.finalize(DEV)
        if kind == "raycast":
            import warnings

            pos, d, far = _camera(case)
            with warnings.catch_warnings():
                warnings.simplefilter("ignore")
                cam = nsph.sensors.SensorRaycast(model, pos, d, (0.0, 0.0, 1.0), 1.0, case["width"], case["height"],
                                                 max_distance=far)
            return dict(kind=kind, sensor=cam, s0=model.state())
        st = dict(kind=kind, model=model, s0=model.state(), s1=model.state(), dt=case["dt"])
        if kind == "contact":
            st["solver"] = SolverSemiImplicit(model)
        else:
            st["solver"] = SolverXPBD(model, iterations=case["iters"])
            st["contacts"] = model.contacts()
        return st
    x, v, flags, f = _fluid(case, seed)
    if case.get("fields"):
        SolverSPH.register_custom_attributes(b)
    b.add_particles(pos=x, vel=v, mass=np.full(len(x), 1000.0 * case["s"] ** 3), flags=flags)
    model = b.finalize(DEV)
    solver = SolverSPH(model, _config(case))
    s0, s1 = model.state(), model.state()
    if f is not None:
        s0.particle_f.copy_(torch.from_numpy(f))
    if kind == "rollout":
        rng = _rng(seed, 4)
        gx, gv = (torch.from_numpy(rng.standard_normal(x.shape, dtype=np.float32)).to(DEV) for _ in range(2))
        eos_b = torch.tensor([_B], dtype=torch.float32, device=DEV, requires_grad=True)
        return dict(kind=kind, solver=solver, x=s0.particle_q.clone().requires_grad_(True),
                    v=s0.particle_qd.clone().requires_grad_(True), b=eos_b, gx=gx, gv=gv, steps=case["steps"],
                    every=case["every"], dt=case["dt"])
    if kind == "surrogate":
        from newton_sph_dev_b200.solvers.sph_surrogate import SurrogateModel, SurrogateSPH

        net = SurrogateModel.pretrained(DEV)
        # the threshold is far above what these states give, so that every call is a surrogate step
        return dict(kind=kind, solver=SurrogateSPH(solver, net, substeps=4, threshold=10.0), s0=s0, s1=s1,
                    dt=case["dt"])
    return dict(kind="sph", solver=solver, s0=s0, s1=s1, dt=case["dt"], fields=bool(case.get("fields")))


def run(state):
    kind = state["kind"]
    if kind == "sph":
        s1 = state["s1"]
        state["solver"].step(state["s0"], s1, None, None, state["dt"])
        out = [s1.particle_q, s1.particle_qd]
        return out + [s1.sph.density, s1.sph.pressure] if state.get("fields") else out
    if kind == "rollout":
        from newton_sph_dev_b200.solvers import sph_rollout

        x1, v1 = sph_rollout(state["solver"], state["x"], state["v"], state["steps"], state["dt"], state["b"],
                             checkpoint_every=state["every"])
        grads = torch.autograd.grad([x1, v1], [state["x"], state["v"], state["b"]], [state["gx"], state["gv"]])
        return [x1.detach(), v1.detach(), *grads]
    if kind == "surrogate":
        state["solver"].step(state["s0"], state["s1"], state["dt"])
        return [state["s1"].particle_q, state["s1"].particle_qd]
    if kind == "contact":
        model, s0, s1 = state["model"], state["s0"], state["s1"]
        model.particle_grid.build(s0.particle_q, 2.0 * model.particle_max_radius + model.particle_cohesion)
        state["solver"].step(s0, s1, None, None, state["dt"])
        return [s1.particle_q, s1.particle_qd, s0.particle_f]
    if kind == "xpbd":
        model, s0, s1 = state["model"], state["s0"], state["s1"]
        s0.particle_q.copy_(model.particle_q)  # the step overwrites its input: each pass is an episode's first
        s0.particle_qd.copy_(model.particle_qd)
        model.collide(s0, state["contacts"])
        state["solver"].step(s0, s1, None, state["contacts"], state["dt"])
        return [s1.particle_q, s1.particle_qd]
    if kind == "raycast":
        state["sensor"].update(state["s0"], include_particles=True)
        return [state["sensor"].get_depth_image()]
    state["grid"].build(state["pts"], state["radius"])
    offsets, ids = state["grid"].query(state["qs"], state["radius"])
    # the sorted order is a view of the grid's own memory: a copy outlives the grid
    return [state["grid"].point_ids.clone(), offsets, ids]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
NEIGHBOURS = 30  # neighbours of a particle within h = 2 spacings, at rest density
STEP_FLOPS = NEIGHBOURS * 60  # a kernel value, its gradient and the sums for each
STEP_BYTES = 24 + 16 + 24  # x, v; mass, inverse mass, flags, world; the new x, v


def work(case):
    kind = case["kind"]
    if kind == "hashgrid":
        per_cell = case["n"] / max(1.0, min(case["extent"] / case["radius"], case["dim"]) ** 3)
        cand = case["q"] * 27 * per_cell
        return {"bytes": case["n"] * 16 + case["q"] * 20 + cand * 4, "flops": case["n"] * 6}
    if kind == "worlds":
        n = case["worlds"] * (16384 - 256) / math.log(16384 / 256)  # the mean of the log-uniform sizes
        return {"bytes": n * STEP_BYTES, "flops": n * STEP_FLOPS}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "rollout":
        return {"bytes": n * 72, "flops": n * STEP_FLOPS * case["steps"] * 4}
    if kind == "surrogate":
        return {"bytes": n * STEP_BYTES, "flops": n * (STEP_FLOPS * 1.5 + 2 * (16 * 64 + 64 * 64 + 64 * 3))}
    if kind == "contact":
        return {"bytes": n * (24 + 16 + 24 + 12), "flops": n * (18 * 10 + 6 * 40)}
    if kind == "xpbd":
        return {"bytes": n * (24 + 16 + 24), "flops": n * case["iters"] * (18 * 10 + 6 * 50)}
    if kind == "raycast":
        return {"bytes": n * 16 + case["width"] * case["height"] * 4, "flops": case["width"] * case["height"] * 200}
    return {"bytes": n * (STEP_BYTES + (12 if case.get("force") else 0) + (8 if case.get("fields") else 0)),
            "flops": n * STEP_FLOPS}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
RHO0, C0, GAMMA, XSPH = 1000.0, 20.0, 7, 0.01
_B = RHO0 * C0 ** 2 / GAMMA


def _d(a):
    return torch.as_tensor(np.asarray(a)).to(DEV, torch.float64)


class _Pairs:
    """The pairs (i, j), i != j, closer than `reach` (a number, or one per
    particle with `group` keeping different groups apart)."""

    def __init__(self, x, reach, group=None, active=None):
        self.x, self.reach = x, reach
        c = torch.floor(x / (reach[:, None] if torch.is_tensor(reach) else reach)).to(torch.int64) + 4
        self.m = int(c.max()) + 8
        key = (c[:, 2] * self.m + c[:, 1]) * self.m + c[:, 0]
        self.key = key if group is None else key + group.to(torch.int64) * self.m ** 3
        ids = torch.arange(len(x), device=x.device) if active is None else torch.nonzero(active).reshape(-1)
        self.who = ids
        order = torch.argsort(self.key[ids])
        self.ids, self.sorted = ids[order], self.key[ids][order]

    def __iter__(self):
        x = self.x
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    k = self.key[self.who] + (dz * self.m + dy) * self.m + dx
                    lo = torch.searchsorted(self.sorted, k)
                    cnt = torch.searchsorted(self.sorted, k, right=True) - lo
                    i = torch.repeat_interleave(self.who, cnt)
                    first = torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
                    j = self.ids[torch.repeat_interleave(lo, cnt) + torch.arange(len(i), device=x.device) - first]
                    d = x[i] - x[j]
                    reach = self.reach[i] if torch.is_tensor(self.reach) else self.reach
                    near = ((d * d).sum(1) < reach * reach) & (i != j)
                    yield i[near], j[near]


def _w(q, sigma):
    t = (1 - q).clamp(min=0)
    return sigma * torch.where(q <= 0.5, 6 * q * q * (q - 1) + 1, 2 * t ** 3)


def _f(q, r, sigma, h):
    """(dW/dr)/r."""
    return torch.where(q <= 0.5, 6 * sigma / (h * h) * (3 * q - 2), -6 * sigma / h * (1 - q).clamp(min=0) ** 2 / r)


class _Fluid64:
    """The WCSPH sums of one state in 64 bits."""

    def __init__(self, h, mass, active=None, group=None):
        self.h, self.m, self.active, self.group = h, mass, active, group
        self.sigma = 8.0 / (math.pi * h ** 3)

    def _of(self, a, i):
        return a[i] if torch.is_tensor(a) and a.dim() else a

    def pairs(self, x):
        with torch.no_grad():
            return list(_Pairs(x, self.h, self.group, self.active))

    def density(self, x, pairs):
        rho = self.m * self.sigma
        if not torch.is_tensor(rho) or not rho.dim():
            rho = torch.full((len(x),), float(rho), dtype=torch.float64, device=x.device)
        if self.active is not None:
            rho = rho * self.active
        for i, j in pairs:
            r = (x[i] - x[j]).norm(dim=1)
            h = self._of(self.h, i)
            rho = rho.index_add(0, i, self._of(self.m, j) * _w(r / h, self._of(self.sigma, i)))
        return rho

    def pressure(self, rho, eos_b):
        return (eos_b * ((rho / RHO0) ** GAMMA - 1)).clamp(min=0)

    def sums(self, x, v, rho, p, pairs, extra=None):
        """Acceleration and XSPH sum (with the surrogate's moments into extra)."""
        live = rho > 0
        safe = torch.where(live, rho, torch.ones_like(rho))
        p2, mor = p / safe ** 2, self.m / safe
        a, dv = torch.zeros_like(x), torch.zeros_like(x)
        for i, j in pairs:
            d = x[i] - x[j]
            r = d.norm(dim=1)
            h, sg = self._of(self.h, i), self._of(self.sigma, i)
            w, f = _w(r / h, sg), _f(r / h, r, sg, h)
            a = a.index_add(0, i, (-self._of(self.m, j) * (p2[i] + p2[j]) * f)[:, None] * d)
            c = mor[j] * w
            rv = v[j] - v[i]
            dv = dv.index_add(0, i, c[:, None] * rv)
            if extra is not None:
                extra["sw"].index_add_(0, i, c)
                extra["mx"].index_add_(0, i, -c[:, None] * d)
                extra["m2"].index_add_(0, i, c * r * r)
                extra["div"].index_add_(0, i, mor[j] * f * (rv * d).sum(1))
        return a, dv

    def advance(self, x, v, a, dv, dt, box, f=None, inv_mass=None):
        g = torch.tensor([0.0, 0.0, -9.81], dtype=torch.float64, device=x.device)
        acc = a + g if f is None else a + f * inv_mass + g
        v1 = v + acc * dt + XSPH * dv
        x1 = x + v1 * dt
        lo, hi = x1 < 0, x1 > box
        v1 = torch.where(lo, v1.clamp(min=0), torch.where(hi, v1.clamp(max=0), v1))
        x1 = torch.where(lo, torch.zeros_like(x1), torch.where(hi, box.expand_as(x1), x1))
        if self.active is not None:
            keep = self.active[:, None]
            x1, v1 = torch.where(keep, x1, x), torch.where(keep, v1, v)
        return x1, v1

    def step(self, x, v, dt, box, eos_b=_B, f=None, inv_mass=None):
        pairs = self.pairs(x)
        rho = self.density(x, pairs)
        p = self.pressure(rho, eos_b)
        if self.active is not None:
            p = p * self.active
        a, dv = self.sums(x, v, rho, p, pairs)
        return (*self.advance(x, v, a, dv, dt, box, f, inv_mass), rho, p)


def _f32(v):
    return float(np.float32(v))


def exact(case, seed):
    kind = case["kind"]
    if kind == "hashgrid":
        return None  # whole numbers
    if kind == "worlds":
        ws = _worlds(case, seed)
        x = _d(np.concatenate([w[0] for w in ws]))
        size = torch.tensor([len(w[0]) for w in ws], device=x.device)
        per = lambda vals: torch.repeat_interleave(_d(np.array(vals)), size)  # noqa: E731
        group = torch.repeat_interleave(torch.arange(len(ws), device=x.device), size)
        fl = _Fluid64(per([_f32(2 * s) for _, s in ws]), per([_f32(1000.0 * s ** 3) for _, s in ws]), group=group)
        box = torch.full((1, 3), WORLD_BOX, dtype=torch.float64, device=x.device)
        return list(fl.step(x, torch.zeros_like(x), _f32(case["dt"]), box)[:2])
    if kind == "raycast":
        return [_exact_depth(case, seed)]
    if kind in ("contact", "xpbd"):
        return _exact_spheres(case, seed)
    x, v, flags, f = _fluid(case, seed)
    x, v = _d(x), _d(v)
    m = _f32(1000.0 * case["s"] ** 3)
    h = _f32(2 * case["s"])
    active = None if flags.all() else _d(flags) > 0
    box = _d(np.array([[_f32(case["bx"]), _f32(case["by"]), _f32(case["bz"])]]))
    dt = _f32(case["dt"])
    fl = _Fluid64(h, m, active)
    if kind == "rollout":
        rng = _rng(seed, 4)
        gx, gv = (_d(rng.standard_normal(tuple(x.shape), dtype=np.float32)) for _ in range(2))
        b = torch.tensor([_f32(_B)], dtype=torch.float64, device=x.device)
        states = [(x, v)]
        for _ in range(case["steps"]):
            states.append(fl.step(*states[-1], dt, box, b)[:2])
        gb = torch.zeros_like(b)
        for xs, vs in reversed(states[:-1]):
            ins = [t.detach().requires_grad_(True) for t in (xs, vs, b)]
            outs = fl.step(ins[0], ins[1], dt, box, ins[2])[:2]
            gx, gv, g = torch.autograd.grad(outs, ins, [gx, gv])
            gb += g
        return [*states[-1], gx, gv, gb]
    if kind == "surrogate":
        return _exact_surrogate(case, fl, x, v, h, m, box)
    f = None if f is None else _d(f)
    x1, v1, rho, p = fl.step(x, v, dt, box, f=f, inv_mass=float(np.float32(1.0) / np.float32(m)))
    return [x1, v1, rho, p] if case.get("fields") else [x1, v1]


def _exact_surrogate(case, fl, x, v, h, m, box):
    from pathlib import Path

    path = Path(os.getcwd()) / "newton_sph_dev_b200" / "surrogate_weights.npz"
    buf = _d(np.load(path, allow_pickle=False)["buf"])
    w1, b1 = buf[0:1024].view(16, 64), buf[1024:1088]
    w2, b2 = buf[1088:5184].view(64, 64), buf[5184:5248]
    w3, b3 = buf[5248:5440].view(64, 3), buf[5440:5443]
    pairs = fl.pairs(x)
    rho = fl.density(x, pairs)
    p = fl.pressure(rho, _B)
    n = len(x)
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device=x.device)  # noqa: E731
    e = dict(sw=z(n), mx=z(n, 3), m2=z(n), div=z(n))
    a, dv = fl.sums(x, v, rho, p, pairs, e)
    c2 = _B * GAMMA / RHO0
    ah = a * h / c2
    feat = torch.cat([(rho / RHO0)[:, None], (rho / RHO0 - 1)[:, None], e["mx"] / h, dv / math.sqrt(c2), ah,
                      (e["m2"] / h ** 2)[:, None], (e["sw"] + m / rho * fl.sigma)[:, None],
                      (e["div"] * h / math.sqrt(c2))[:, None], (p / (RHO0 * c2))[:, None],
                      ah.norm(dim=1, keepdim=True)], 1)
    silu = torch.nn.functional.silu
    y = silu(silu(((feat - buf[5448:5464]) * buf[5464:5480]) @ w1 + b1) @ w2 + b2) @ w3 + b3
    da = (y * buf[5484:5487] + buf[5480:5483]) * (c2 / h)
    return list(fl.advance(x, v, a + da, dv, _f32(4 * case["dt"]), box))


def _friction_and_normal(x, v, i, j):
    d = x[i] - x[j]
    dist = d.norm(dim=1)
    n = d / dist[:, None]
    rv = v[i] - v[j]
    vn = (n * rv).sum(1)
    vt = rv - n * vn[:, None]
    lt = vt.norm(dim=1)
    return dist, n, vn, vt / torch.where(lt > 0, lt, torch.ones_like(lt))[:, None], lt


def _exact_spheres(case, seed):
    x, v, rad = (_d(a) for a in _spheres(case, seed))
    dt = _f32(case["dt"])
    g = torch.tensor([0.0, 0.0, -9.81], dtype=torch.float64, device=x.device)
    reach = 2.0 * float(rad.max()) * 1.02
    if case["kind"] == "contact":
        f = torch.zeros_like(x)
        for i, j in _Pairs(x, reach):
            dist, n, vn, t, lt = _friction_and_normal(x, v, i, j)
            err = dist - rad[i] - rad[j]
            fn = err * 1e3 + vn.clamp(max=0) * 1e2
            ft = torch.minimum(lt * 1e2, 0.5 * fn.abs())
            c = -n * fn[:, None] - t * ft[:, None]
            f.index_add_(0, i, torch.where((err <= 0)[:, None], c, torch.zeros_like(c)))
        v1 = v + (f + g) * dt
        return [x + v1 * dt, v1, f]
    # the contacts with the ground come from the state before the step
    ground = x[:, 2] < 0.01 + rad
    vel = v + g * dt
    pos = x + vel * dt
    pairs = [torch.cat(t) for t in zip(*_Pairs(pos, reach * 1.25))]
    for _ in range(case["iters"]):
        dlt = torch.zeros_like(x)
        c = pos[:, 2] - rad
        vt = vel * torch.tensor([1.0, 1.0, 0.0], dtype=torch.float64, device=x.device)
        lt = vt.norm(dim=1)
        lf = torch.maximum(0.5 * c, -lt * dt)
        one = vt / torch.where(lt > 0, lt, torch.ones_like(lt))[:, None] * lf[:, None]
        one[:, 2] -= c
        dlt += torch.where((ground & (c <= 0))[:, None], one * 0.9, torch.zeros_like(one))
        i, j = pairs
        dist, n, vn, t, lt = _friction_and_normal(pos, vel, i, j)
        err = dist - rad[i] - rad[j]
        lf = torch.maximum(0.5 * err, -lt * dt)
        one = (t * lf[:, None] - n * err[:, None]) / 2.0
        part = torch.zeros_like(x).index_add_(0, i, torch.where((err <= 0)[:, None], one, torch.zeros_like(one)))
        pos = pos + dlt + part * 0.9
        vel = (pos - x) / dt
    return [pos, vel]


def _exact_depth(case, seed):
    """Nearest hit of every pixel's ray, by projecting each sphere onto the
    pixels that it may cover."""
    x, _, rad = (_d(a) for a in _spheres(case, seed))
    pos, d, far = _camera(case)
    w, h = case["width"], case["height"]
    pos, d = np.float32(pos), np.float32(d)
    d = d / np.linalg.norm(d)
    right = np.cross(d, np.array([0, 0, 1], np.float32))
    right = right / np.linalg.norm(right)
    up = np.cross(right, d)
    up = up / np.linalg.norm(up)
    o, fwd, rt, upv = _d(pos), _d(d), _d(right), _d(up)
    scale = _f32(math.tan(0.5))
    aspect = _f32(w / h)
    rel = x - o
    depth_z = rel @ fwd
    px = ((rel @ rt) / depth_z / (scale * aspect) + 1) * 0.5 * w - 0.5
    py = (1 - (rel @ upv) / depth_z / scale) * 0.5 * h - 0.5
    k = int(math.ceil(float((rad / (depth_z - rad)).max()) / scale * 0.5 * h * 1.5)) + 1
    out = torch.full((h * w,), math.inf, dtype=torch.float64, device=x.device)
    cx, cy = torch.round(px).long(), torch.round(py).long()
    for oy in range(-k, k + 1):
        for ox in range(-k, k + 1):
            ix, iy = cx + ox, cy + oy
            ok = (ix >= 0) & (ix < w) & (iy >= 0) & (iy < h)
            nx = ((2.0 * ix[ok] + 1) / w - 1) * scale * aspect
            ny = (1 - (2.0 * iy[ok] + 1) / h) * scale
            ray = nx[:, None] * rt + ny[:, None] * upv + fwd
            ray = ray / ray.norm(dim=1, keepdim=True)
            oc = -rel[ok]
            b = (ray * oc).sum(1)
            disc = b * b - ((oc * oc).sum(1) - rad[ok] ** 2)
            t = -b - disc.clamp(min=0).sqrt()
            hit = (disc >= 0) & (t >= 0) & (t < far)
            out.scatter_reduce_(0, (iy[ok] * w + ix[ok])[hit], t[hit], "amin")
    return torch.where(torch.isinf(out), torch.full_like(out, -1.0), out).view(h, w)
