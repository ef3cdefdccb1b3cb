"""Small scenes take their own kernels (a build by counting comparisons, eight
lanes per particle in the density pass, four in the force pass); the latter
two not where a launch shape is set. Their results are those of the large-scene kernels and of the
oracle, at the edges of each range."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_hashgrid import _grid_arrays, _points
from test_gpu_tiles import NAMES, _cloud, _scene

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("dims", [(128, 128, 128), (37, 29, 31), (16, 16, 16), (2, 1, 1)])
def test_small_builds_match_oracle(oracle_mod, dims):
    """Sizes around a warp's and a warp's loads, around the range and around the
    largest predecessor, in turn on one grid with builds of the other kinds
    (each clears its predecessor's cells)."""
    from newton_sph_dev_b200 import HashGrid

    grid = HashGrid(*dims, device=DEV)
    for seed, n in enumerate((1, 31, 32, 33, 70000, 1024, 1025, 65537, 4095, 4096, 65536, 4097, 8191, 20000, 8192, 8193)):
        pts = _points(n, seed, special=seed % 2 == 0)
        grid.build(torch.from_numpy(pts).to(DEV), 0.037)
        torch.cuda.synchronize()
        got = _grid_arrays(grid)
        ref = oracle_mod.grid_build(pts, 0.037, dims)
        for k in ref:
            np.testing.assert_array_equal(got[k], ref[k], err_msg=f"n={n}: {k}")


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("worlds", [False, True])
def test_small_and_large_scene_kernels_agree(name, worlds):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    x, kw = _scene(name)
    n = len(x)
    rng = np.random.default_rng(7)
    flags = np.ones(n, np.int32)
    if n > 40:
        flags[rng.random(n) < 0.05] = 0
    b = nsph.ModelBuilder()
    SolverSPH.register_custom_attributes(b)
    cfg = SolverSPH.Config(smoothing_length=0.02, **kw)
    if worlds:
        b.begin_world()
    b.add_particles(pos=x, vel=rng.normal(0, 0.1, x.shape).astype(np.float32), mass=np.full(n, 1e-3), flags=flags)
    if worlds:
        b.end_world()
        b.begin_world()
        y = _cloud(77, 0.05, 50)
        b.add_particles(pos=y, vel=np.zeros_like(y), mass=np.full(len(y), 1e-3))
        b.end_world()
        cfg = [cfg, SolverSPH.Config(smoothing_length=0.013, grid_dims=(32, 32, 32))]
    model = b.finalize(DEV)
    out = []
    for launch in (None, (256, 0), (128, 0)):
        solver = SolverSPH(model, cfg)
        if launch:
            solver.set_launch(*launch)
        s0, s1 = model.state(), model.state()
        solver.step(s0, s1, None, None, 1e-5)
        out.append([t.cpu().numpy() for t in (s1.sph.density, s1.sph.pressure, s1.particle_q, s1.particle_qd)])
    for other in out[1:]:
        for a, c in zip(out[0], other):
            np.testing.assert_array_equal(a, c)
