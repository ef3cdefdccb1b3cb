"""The contact kernels' bounded candidate test and waiting list, bit-exact
against the oracle: piles with more contacts than a thread's waiting slots,
contacts at the bound itself (touching lattices), negative and large
cohesion, radii of zero and of very different sizes, and coincident
particles."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DIMS = (64, 64, 64)


def _scene(name):
    rng = np.random.default_rng(3)
    if name == "touching":  # distances of exactly r_i + r_j and one rounding off
        g = np.stack(np.meshgrid(*[np.arange(11)] * 3, indexing="ij"), -1).reshape(-1, 3)
        x = (g * np.float32(0.01) + np.float32(0.3)).astype(np.float32)
        return x, np.full(len(x), 0.005, np.float32), 0.0
    if name == "pile":  # ~120 contacts each
        return (rng.random((700, 3)) * 0.05 + 0.2).astype(np.float32), np.full(700, 0.01, np.float32), 0.0
    x = rng.random((4000, 3)).astype(np.float32)
    r = rng.uniform(0.004, 0.02, 4000).astype(np.float32)
    if name == "negative_cohesion":
        return x, r, -0.004
    if name == "large_cohesion":
        return x, r, 0.03
    if name == "mixed_radii":
        r = (0.03 * 10 ** rng.uniform(-4, 0, 4000)).astype(np.float32)
        r[::7] = 0.0
        return x, r, 0.001
    if name == "coincident":
        x[1::2] = x[0::2]
        return x, r, 0.0
    raise KeyError(name)


@pytest.mark.parametrize("name", ["touching", "pile", "negative_cohesion", "large_cohesion", "mixed_radii",
                                  "coincident"])
def test_forces_and_deltas(oracle_mod, name):
    from newton_sph_dev_b200 import HashGrid, _lib

    x, r, cohesion = _scene(name)
    n = len(x)
    rng = np.random.default_rng(4)
    v = rng.normal(0, 0.5, (n, 3)).astype(np.float32)
    flags = (rng.random(n) > 0.05).astype(np.int32)
    w = rng.uniform(0.5, 2.0, n).astype(np.float32)
    rmax = float(r.max())
    gr = float(np.float32(2 * rmax + max(cohesion, 0.0)))
    T = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    xt, vt, rt, ft, wt = T(x), T(v), T(r), T(flags), T(w)
    g = HashGrid(*DIMS, device=DEV)
    g.build(xt, gr)
    L, stream = _lib.load(), _lib.stream_handle(torch.device(DEV))
    f = torch.full((n, 3), 7.0, device=DEV)
    p = _lib.NsphContactParams(1000.0, 100.0, 100.0, 0.5, cohesion, rmax)
    _lib.check(L.nsph_particle_contact_forces(g.id, ctypes.byref(p), n, xt.data_ptr(), vt.data_ptr(), rt.data_ptr(),
                                              ft.data_ptr(), f.data_ptr(), stream), "forces")
    ref = oracle_mod.particle_contact_forces(x, v, r, flags, gr, DIMS, 1000.0, 100.0, 100.0, 0.5, cohesion, rmax,
                                             f_init=np.full((n, 3), 7.0, np.float32))
    np.testing.assert_array_equal(f.cpu().numpy(), ref)
    init = rng.normal(0, 1e-3, (n, 3)).astype(np.float32)
    d = T(init.copy())
    _lib.check(L.nsph_particle_contact_deltas(g.id, n, xt.data_ptr(), vt.data_ptr(), wt.data_ptr(), rt.data_ptr(),
                                              ft.data_ptr(), 0.5, cohesion, rmax, 1e-3, 0.8, d.data_ptr(), stream),
               "deltas")
    ref = oracle_mod.particle_contact_deltas(x, v, w, r, flags, gr, DIMS, 0.5, cohesion, rmax, 1e-3, 0.8, init)
    np.testing.assert_array_equal(d.cpu().numpy(), ref)
