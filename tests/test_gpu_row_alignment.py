"""Rows of three floats are read and written as one 8-byte and one 4-byte
access, chosen by the row's address: states whose arrays start at an odd
multiple of four bytes give the same results as aligned ones."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _shifted(t, rows):
    """The same values in a view that starts `rows` rows into its buffer."""
    buf = torch.full((t.shape[0] + rows, 3), float("nan"), device=t.device)
    buf[rows:] = t
    return buf[rows:]


def _model(n, sph):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    rng = np.random.default_rng(n)
    b = nsph.ModelBuilder()
    if sph:
        SolverSPH.register_custom_attributes(b)
    side = 0.01 * n ** (1 / 3)
    b.add_particles(pos=(rng.random((n, 3)) * side + 0.02).astype(np.float32),
                    vel=rng.normal(0, 0.1, (n, 3)).astype(np.float32), mass=np.full(n, 1e-3), radius=np.full(n, 0.005))
    return b.finalize(DEV)


@pytest.mark.parametrize("n", [1, 33, 3000, 30000])
@pytest.mark.parametrize("kind", ["sph", "semi_implicit", "xpbd", "gradient"])
def test_shifted_rows(n, kind):
    from newton_sph_dev_b200.solvers import SolverSemiImplicit, SolverSPH, SolverXPBD
    from newton_sph_dev_b200.solvers.sph_diff import sph_rollout

    model = _model(n, kind in ("sph", "gradient"))
    if kind in ("sph", "gradient"):
        solver = SolverSPH(model, SolverSPH.Config(smoothing_length=0.02, box_lo=(0.0,) * 3, box_hi=(0.6,) * 3))
    elif kind == "xpbd":
        solver = SolverXPBD(model, iterations=3)
    else:
        solver = SolverSemiImplicit(model)
    results = []
    for rows in (0, 1):
        s0, s1 = model.state(), model.state()
        s0.particle_f.copy_(torch.linspace(-1e-3, 1e-3, 3 * n, device=DEV).reshape(n, 3))
        if kind == "gradient":
            x, v = (_shifted(t, rows).requires_grad_() for t in (s0.particle_q, s0.particle_qd))
            xt, vt = sph_rollout(solver, x, v, 3, 1e-4, checkpoint_every=2)
            gx, gv = torch.autograd.grad((xt * _shifted(torch.cos(xt.detach()), rows)).sum() + vt.square().sum(), (x, v))
            results.append([t.detach().cpu().numpy() for t in (xt, vt, gx, gv)])
            continue
        for s in (s0, s1):
            for name in ("particle_q", "particle_qd", "particle_f"):
                setattr(s, name, _shifted(getattr(s, name), rows))
        if kind == "semi_implicit" and model.particle_grid is not None:
            model.particle_grid.build(s0.particle_q, 0.012)
        solver.step(s0, s1, None, model.contacts() if kind == "xpbd" else None, 1e-4)
        results.append([t.cpu().numpy() for t in (s1.particle_q, s1.particle_qd)])
    for a, c in zip(*results):
        np.testing.assert_array_equal(a, c)
