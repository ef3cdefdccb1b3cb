"""SolverSPH.autotune on a scene small enough for the several-threads kernels,
which an explicit launch shape turns off: the default is among what it times."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("worlds", [False, True])
def test_the_default_can_win(worlds):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    rng = np.random.default_rng(0)
    b = nsph.ModelBuilder()
    SolverSPH.register_custom_attributes(b)
    for _ in range(2 if worlds else 1):
        if worlds:
            b.begin_world()
        b.add_particles(pos=(rng.random((2000, 3)) * 0.12).astype(np.float32), vel=np.zeros((2000, 3), np.float32),
                        mass=np.full(2000, 1e-3))
        if worlds:
            b.end_world()
    model = b.finalize("cuda:0")
    cfg = SolverSPH.Config(smoothing_length=0.02, box_lo=(0.0,) * 3, box_hi=(0.2,) * 3)
    solver = SolverSPH(model, [cfg, cfg] if worlds else cfg)
    s0, s1 = model.state(), model.state()
    res = solver.autotune(s0, s1, 1e-5)
    assert (0, -1) in res and len(res) == 12
    assert res["best"] == min((k for k in res if k != "best"), key=res.get)
    assert res[res["best"]] <= res[(0, -1)]
    assert solver.launch == res["best"]
