"""The large scenes' kernels on scenes small enough for the oracles. A launch
shape set by the caller takes them at every size (small scenes otherwise have
kernels with several lanes per particle): the neighbour tiles and the force
walk on every edge scene of test_gpu_tiles, bit-exact; a scene whose warps
take several groups of particles in turn; the tolerance arithmetic; the
adjoint, rollout and segment checks of test_gpu_adjoint; and a segment whose
neighbour lists overflow in some of its steps only."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import test_gpu_adjoint as adjoint
import test_gpu_tiles as tiles
from test_gpu_tiles import DEV, NAMES, _cloud, _scene

pytestmark = pytest.mark.gpu

SHAPES = [(256, 0), (64, 1)]


@pytest.fixture
def shaped(monkeypatch, request):
    """Every solver made in the test has the launch shape `request.param`."""
    from newton_sph_dev_b200.solvers import SolverSPH

    init = SolverSPH.__init__

    def with_shape(self, *args, **kwargs):
        init(self, *args, **kwargs)
        if request.param:
            self.set_launch(*request.param)

    monkeypatch.setattr(SolverSPH, "__init__", with_shape)
    return request.param


@pytest.mark.parametrize("shaped", SHAPES, indirect=True)
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("worlds", [False, True])
def test_tiles_equal_oracle(oracle_mod, shaped, name, worlds):
    tiles.test_step_equals_oracle(oracle_mod, name, worlds)


def _strides():
    """24,000 particles: three strides of 148 blocks of 64 threads, with runs
    that wrap around the grid, a cluster whose lists overflow, particles on cell
    borders, inactive and non-finite ones."""
    x = _cloud(24000, 0.3, 21, lo=-0.1)
    x[:300] = _cloud(300, 0.012, 22, lo=0.05)
    x[5000:8000:3] = np.round(x[5000:8000:3] / 0.02).astype(np.float32) * np.float32(0.02)
    x[9000, 0], x[15000, 1], x[21000, 2] = np.nan, np.inf, -3e38
    return x, dict(grid_dims=(18, 16, 17))


@pytest.mark.parametrize("shaped", [None, (64, 1), (32, 2), (256, 0)], indirect=True)
@pytest.mark.parametrize("worlds", [False, True])
def test_warps_that_take_several_groups(oracle_mod, shaped, worlds, monkeypatch):
    monkeypatch.setattr(tiles, "_scene", lambda name: _strides())
    tiles.test_step_equals_oracle(oracle_mod, "strides", worlds)


@pytest.mark.parametrize("shaped", [None, (256, 0), (64, 1)], indirect=True)
@pytest.mark.parametrize("name", NAMES + ["strides"])
def test_tolerance_arithmetic(oracle_mod, shaped, name):
    """Densities against the fp32 oracle. Per neighbour, of the kernel's value
    at zero: 4e-7 of q (a reciprocal square root of 2 ulp and two roundings)
    times at most 0.67, and six roundings on either side: below 1e-6 in all; and
    the rounding of each partial sum on either side. A neighbour that is missed
    or added inside the support is far outside that."""
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    x, kw = _strides() if name == "strides" else _scene(name)
    n = len(x)
    flags = np.ones(n, np.int32)
    flags[3::17] = 0
    cfg = SolverSPH.Config(smoothing_length=0.02, arithmetic="fast", **kw)
    b = nsph.ModelBuilder()
    SolverSPH.register_custom_attributes(b)
    b.add_particles(pos=x, vel=np.zeros_like(x), mass=np.full(n, 1e-3), flags=flags)
    model = b.finalize(DEV)
    solver = SolverSPH(model, cfg)
    s0, s1 = model.state(), model.state()
    solver.step(s0, s1, None, None, 1e-5)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    consts = cfg.constants(1e-5, model.particle_max_velocity)
    r = oracle_mod.sph_step(consts, solver.grid_dims, x, np.zeros_like(x), host(model.particle_mass),
                            host(model.particle_inv_mass), flags, np.zeros(n, np.int32), host(model.gravity)[:1],
                            v_out_init=np.zeros_like(x), precision="f32")
    count = np.diff(oracle_mod.sph_neighbors(consts["f32"], solver.grid_dims, x, flags)[0])
    bound = 1e-6 * (1 + count) * (1e-3 * consts["f32"]["sigma"]) + 1.2e-7 * count * r["rho"]
    off = np.abs(host(s1.sph.density).astype(np.float64) - r["rho"])
    assert np.all(off <= bound)


@pytest.mark.parametrize("shaped", SHAPES, indirect=True)
@pytest.mark.parametrize("clamp", [True, False])
def test_step_adjoint(oracle_mod, shaped, clamp):
    adjoint.test_step_adjoint_matches_fp64_oracle(oracle_mod, clamp)


@pytest.mark.parametrize("shaped", SHAPES, indirect=True)
@pytest.mark.parametrize("clamp", [True, False])
def test_rollout_gradient(oracle_mod, shaped, clamp):
    adjoint.test_rollout_gradient_matches_fp64_and_central_differences(oracle_mod, clamp)


@pytest.mark.parametrize("shaped", SHAPES, indirect=True)
@pytest.mark.parametrize("check", [adjoint.test_adjoint_in_place_and_deterministic,
                                   adjoint.test_checkpointing_does_not_change_gradients,
                                   adjoint.test_segment_tape_equals_recompute_then_reverse])
def test_adjoint_identities(shaped, check):
    check()


@pytest.mark.parametrize("shaped", [None, (256, 0), (64, 1)], indirect=True)
def test_segment_whose_lists_overflow_in_some_steps(shaped):
    """A cluster that expands through the lists' 64 slots beside a block: the
    segment's gradients are those of the recomputed rollout, bit for bit, with a
    tape that another scene has filled before."""
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    s, dt, steps = 0.01, 1e-4, 8
    rng = np.random.default_rng(4)
    g = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3)
    block = (g + 0.5) * s + rng.uniform(-0.1 * s, 0.1 * s, g.shape) + 0.05
    d = rng.normal(size=(120, 3))
    cluster = d / np.linalg.norm(d, axis=1)[:, None] * (0.009 * rng.random((120, 1)) ** (1 / 3))
    centre = np.array([0.25, 0.09, 0.1])
    x = np.concatenate([block, cluster + centre]).astype(np.float32)
    v = np.concatenate([rng.normal(0, 0.1, block.shape), 4500.0 * cluster]).astype(np.float32)
    mass = np.concatenate([np.full(len(block), 1000 * s**3), np.full(120, 0.02 * 1000 * s**3)])
    order = rng.permutation(len(x))
    x, v, mass = x[order], v[order], mass[order]
    b = nsph.ModelBuilder()
    b.add_particles(pos=x, vel=v, mass=mass)
    model = b.finalize(DEV)
    cfg = SolverSPH.Config(smoothing_length=2 * s, box_lo=(0.0,) * 3, box_hi=(0.4,) * 3)
    solver = SolverSPH(model, cfg)
    p = solver.step_params(dt)
    n = len(x)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)  # noqa: E731
    x0, v0 = T(x), T(v)
    gx, gv = T(rng.normal(size=x.shape)), T(rng.normal(size=x.shape))

    sx = torch.empty((steps, n, 3), dtype=torch.float32, device=DEV)
    sv = torch.empty_like(sx)
    sx[0].copy_(x0)
    sv[0].copy_(v0)
    solver.rollout_raw(sx[0], sv[0], sx[1:], sv[1:], p, None)
    xa, va, ba = gx.clone(), gv.clone(), torch.zeros(1, device=DEV)
    solver.rollout_backward_raw(sx, sv, p, xa, va, eos_b_grad=ba)
    most = []
    for t in range(steps):
        solver.step_raw(sx[t], sv[t], torch.empty_like(x0), sv[t].clone(), p, None)
        most.append(int(torch.diff(solver.neighbors()[0]).max()))
    assert most[0] > 64 and most[-1] <= 64, most

    # the tape first holds a scene with other cells and lists that all overflow
    other = T((x - 0.5 * x.mean(0)) * 0.3 + 0.1)
    solver.segment_backward_raw(other, v0, steps, p, gx.clone(), gv.clone())
    for _ in range(2):
        xb, vb, bb = gx.clone(), gv.clone(), torch.zeros(1, device=DEV)
        solver.segment_backward_raw(x0, v0, steps, p, xb, vb, eos_b_grad=bb)
        torch.cuda.synchronize()
        assert torch.isfinite(xa).all()
        for a, c in ((xa, xb), (va, vb), (ba, bb)):
            assert torch.equal(a, c)
        # and once with the overflowing steps last: the state runs backwards
        solver.segment_backward_raw(sx[-1], -sv[-1], steps, p, gx.clone(), gv.clone())
