"""The tensor-core neighbour tiles of the density pass and the force pass's
group walk, bit-exact against the fp32 oracle where they can go wrong: warps
of one particle and of a tile plus one, particles scattered over many rows,
stencils that wrap around the grid or span it, cells much narrower and much
wider than the kernel support, coordinates whose cells the 2^20 origin
clamps, particles exactly on cell borders, lists that overflow and
non-finite positions; and the force terms' square root over every mantissa.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _cloud(n, extent, seed=0, lo=0.0):
    return (np.random.default_rng(seed).random((n, 3)) * extent + lo).astype(np.float32)


def _scene(name):
    """(positions, config arguments)"""
    h = 0.02
    box = dict(box_lo=(0.0, 0.0, 0.0), box_hi=(0.4, 0.4, 0.4))
    if name.startswith("n="):
        return _cloud(int(name[2:]), 0.06), box
    if name == "scattered":  # about one particle per row of cells
        return _cloud(3000, 2.0, 1), dict(grid_dims=(100, 100, 100))
    if name == "wraps":  # the block straddles the grid's period on every axis
        return _cloud(2500, 0.12, 2, lo=-0.05), dict(grid_dims=(9, 8, 7))
    if name == "narrow_grid":  # stencils as wide as the grid
        return _cloud(700, 0.1, 3), dict(grid_dims=(4, 3, 5))
    if name == "one_cell":
        return _cloud(300, 0.05, 4), dict(grid_dims=(1, 1, 1))
    if name == "narrow_cells":
        return _cloud(1500, 0.1, 5), dict(cell_width=0.3 * h, **box)
    if name == "wide_cells":
        return _cloud(1500, 0.3, 6), dict(cell_width=2.3 * h, **box)
    if name == "cells_100h":
        return _cloud(400, 3.0, 7), dict(cell_width=100 * h, grid_dims=(16, 16, 16))
    if name == "negative":
        return _cloud(2000, 0.1, 8, lo=-0.35), dict(grid_dims=(64, 64, 64))
    if name == "far":  # cells in the hundreds of thousands: coarse coordinates
        return _cloud(1500, 0.1, 9, lo=9000.0), dict(grid_dims=(64, 64, 64))
    if name == "clamped":  # below the 2^20 origin
        x = _cloud(400, 0.1, 10)
        x[::3] -= np.float32(30000.0)
        return x, dict(grid_dims=(64, 64, 64))
    if name == "borders":  # multiples of h: distances of exactly h, cells by one rounding
        g = np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)
        return (g.astype(np.float32) * np.float32(h / 2) + np.float32(0.06)).astype(np.float32), box
    if name == "border_roundings":
        rng = np.random.default_rng(11)
        x = rng.integers(3, 12, (3000, 3)).astype(np.float32) * np.float32(h)
        x = np.nextafter(x, x + rng.choice([-1.0, 1.0], x.shape).astype(np.float32)).astype(np.float32)
        x[:, 1:] = (x[:, 1:] + rng.random((3000, 2)).astype(np.float32) * np.float32(0.3 * h))
        return x, box
    if name == "overflow":  # far more than the list's 64 slots
        return np.concatenate([_cloud(260, 0.012, 12, lo=0.1), _cloud(500, 0.1, 13, lo=0.1)]), box
    if name == "coincident":
        x = _cloud(300, 0.06, 14)
        x[1::4] = x[0::4][: len(x[1::4])]
        x[2::4] = np.nextafter(x[0::4][: len(x[2::4])], np.float32(1.0))
        return x, box
    if name == "long_runs":  # a line of particles: runs of many chunks
        x = _cloud(1500, 0.004, 15, lo=0.1)
        x[:, 0] = np.linspace(0.02, 0.3, 1500, dtype=np.float32)
        return x, box
    if name == "non_finite":
        x = _cloud(900, 0.08, 16)
        x[5, 0], x[17, 1], x[40, 2] = np.nan, np.inf, -np.inf
        x[77] = 3e38
        return x, box
    raise KeyError(name)


NAMES = ["n=1", "n=2", "n=31", "n=32", "n=33", "n=257", "scattered", "wraps", "narrow_grid", "one_cell",
         "narrow_cells", "wide_cells", "cells_100h", "negative", "far", "clamped", "borders", "border_roundings",
         "overflow", "coincident", "long_runs", "non_finite"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("worlds", [False, True])
def test_step_equals_oracle(oracle_mod, name, worlds):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    x, kw = _scene(name)
    n = len(x)
    rng = np.random.default_rng(99)
    v = rng.normal(0, 0.1, x.shape).astype(np.float32)
    flags = np.ones(n, np.int32)
    if n > 40:
        flags[rng.random(n) < 0.05] = 0
    cfg = SolverSPH.Config(smoothing_length=0.02, **kw)
    b = nsph.ModelBuilder()
    SolverSPH.register_custom_attributes(b)
    if worlds:
        b.begin_world()
    b.add_particles(pos=x, vel=v, mass=np.full(n, 1e-3), flags=flags)
    if worlds:  # a second world in the same warps, at another spacing
        b.end_world()
        b.begin_world()
        y = _cloud(77, 0.05, 50)
        b.add_particles(pos=y, vel=np.zeros_like(y), mass=np.full(len(y), 1e-3))
        b.end_world()
    model = b.finalize(DEV)
    solver = SolverSPH(model, [cfg, SolverSPH.Config(smoothing_length=0.013, grid_dims=(32, 32, 32))]
                       if worlds else cfg)
    dims = solver.world_grid_dims[0] if worlds else solver.grid_dims
    s0, s1 = model.state(), model.state()
    dt = 1e-5
    solver.step(s0, s1, None, None, dt)
    host = lambda t: t.cpu().numpy()[:n]  # noqa: E731
    consts = cfg.constants(dt, model.particle_max_velocity)
    r = oracle_mod.sph_step(consts, dims, x, v, host(model.particle_mass), host(model.particle_inv_mass), flags,
                            np.zeros(n, np.int32), host(model.gravity)[:1], v_out_init=v, precision="f32")
    np.testing.assert_array_equal(host(s1.sph.density), r["rho"])
    np.testing.assert_array_equal(host(s1.sph.pressure), r["p"])
    np.testing.assert_array_equal(host(s1.particle_q), r["x"])
    np.testing.assert_array_equal(host(s1.particle_qd), r["v"])


def test_force_roots_are_correctly_rounded():
    from newton_sph_dev_b200 import _lib

    e = (ctypes.c_int * 6)(0, -7, 7, -50, 49, -13)
    count = ctypes.c_ulonglong(1)
    _lib.check(_lib.load().nsph_debug_root_mismatches(e, 6, ctypes.byref(count)), "sweep")
    assert count.value == 0
