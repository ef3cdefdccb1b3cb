"""The density pass's candidate filter with pairs at the very edge of the
support, at both ends of the longest groups of particles that it takes
(rows of twelve cells) and in cells from a third of the support to several of
it: bit-exact against the fp32 oracle, for the large scenes' kernels."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
H = np.float32(0.02)


def _rows(cell, seed):
    """Rows of 32 particles over twelve cells, most of them at the rows' ends,
    each with a partner at H (1 - 2^-22) or a rounding from it; rows far enough
    apart that a warp is a row with its partners' rows between."""
    rng = np.random.default_rng(seed)
    pts = []
    for iz in range(4):
        for iy in range(4):
            t = np.concatenate([rng.uniform(0, 0.9, 8), rng.uniform(11.1, 12, 8), rng.uniform(0, 12, 16)])
            p = np.stack([t, np.full(32, 2 + 5 * iy) + rng.random(32), np.full(32, 2 + 5 * iz) + rng.random(32)], 1)
            p = (p + [3, 0, 0]) * cell
            e = rng.normal(size=p.shape)
            e[::4] = [1, 0, 0]
            e[1::4] *= [1, 0.05, 0.05]
            e[:8] *= np.sign(e[:8, :1]) * [-1, 1, 1]  # outwards
            e /= np.linalg.norm(e, axis=1)[:, None]
            p = p.astype(np.float32)
            q = (p + e * (float(H) * (1 - 2.0**-22))).astype(np.float32)
            q[5::6] = np.nextafter(q[5::6], p[5::6])
            pts += [p, q]
    return np.concatenate(pts)


@pytest.mark.parametrize("launch", [(256, 0), (64, 1)])
@pytest.mark.parametrize("cells", [0.34, 1.0, 2.3, 4.0])
def test_pairs_at_the_edge(oracle_mod, cells, launch):
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    x = np.concatenate([_rows(cells * float(H), s) for s in (1, 2)])
    n = len(x)
    cfg = SolverSPH.Config(smoothing_length=float(H), cell_width=cells * float(H), grid_dims=(64, 64, 64))
    b = nsph.ModelBuilder()
    SolverSPH.register_custom_attributes(b)
    b.add_particles(pos=x, vel=np.zeros_like(x), mass=np.full(n, 1e-3))
    model = b.finalize(DEV)
    solver = SolverSPH(model, cfg)
    solver.set_launch(*launch)
    s0, s1 = model.state(), model.state()
    solver.step(s0, s1, None, None, 1e-6)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    r = oracle_mod.sph_step(cfg.constants(1e-6, model.particle_max_velocity), solver.grid_dims, x, np.zeros_like(x),
                            host(model.particle_mass), host(model.particle_inv_mass), np.ones(n, np.int32),
                            np.zeros(n, np.int32), host(model.gravity)[:1], v_out_init=np.zeros_like(x),
                            precision="f32")
    np.testing.assert_array_equal(host(s1.sph.density), r["rho"])
    np.testing.assert_array_equal(host(s1.sph.pressure), r["p"])
    np.testing.assert_array_equal(host(s1.particle_q), r["x"])
    np.testing.assert_array_equal(host(s1.particle_qd), r["v"])
