"""The raycast's tree and its shortened march, bit-exact against the oracle's
full march where they can differ: cameras inside the block, spheres that
overlap heavily, marches longer and shorter than a sphere, radii of very
different sizes, grids that alias, truncated marches, outliers far from the
scene, spheres out of range and tiny inputs."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_raycast import _camera, _device_depth

pytestmark = pytest.mark.gpu


def _block(n, spacing, seed, jitter=0.1):
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    return ((g + 0.5 + rng.uniform(-jitter, jitter, g.shape)) * spacing).astype(np.float32)


CASES = {
    # x, r, position, direction, fov, dims, search radius, step, max distance, max steps (0: as needed)
    "inside": lambda: (_block(20, 0.02, 1), 0.006, (0.21, 0.2, 0.19), (1, 0.3, 0.2), 1.4, (128,) * 3, 0, 0.5, 2.0, 0),
    "overlap": lambda: (_block(20, 0.01, 2), 0.03, (0.6, -0.5, 0.4), (-0.5, 0.7, -0.3), 0.7, (128,) * 3, 0, 0.5, 2.0, 0),
    "long_step": lambda: (_block(16, 0.02, 3), 0.01, (0.8, -0.6, 0.5), (-0.7, 0.8, -0.4), 0.6, (64, 50, 33), 0, 3.7,
                          3.0, 0),
    "short_step": lambda: (_block(10, 0.02, 4), 0.01, (0.5, -0.3, 0.4), (-0.4, 0.5, -0.3), 0.5, (32,) * 3, 0, 0.05,
                           1.0, 0),
    "aliases": lambda: (_block(24, 0.02, 5), 0.009, (1.2, -0.9, 0.8), (-0.9, 1.1, -0.5), 0.5, (16, 11, 9), 0, 0.5,
                        4.0, 0),
    "truncated": lambda: (_block(16, 0.02, 6), 0.01, (0.8, -0.6, 0.5), (-0.7, 0.8, -0.4), 0.6, (128,) * 3, 0, 0.5,
                          3.0, 190),
    "wide_search": lambda: (_block(12, 0.02, 7), 0.004, (0.7, -0.5, 0.4), (-0.6, 0.7, -0.3), 0.5, (128,) * 3, 0.02,
                            0.5, 2.0, 0),
    "narrow_search": lambda: (_block(12, 0.02, 8), 0.01, (0.7, -0.5, 0.4), (-0.6, 0.7, -0.3), 0.5, (128,) * 3, 0.003,
                              0.5, 2.0, 0),
    "short_range": lambda: (_block(16, 0.02, 9), 0.01, (0.8, -0.6, 0.5), (-0.7, 0.8, -0.4), 0.8, (128,) * 3, 0, 0.5,
                            0.9, 0),
    "axis": lambda: (_block(16, 0.02, 10, 0.0), 0.01, (0.16, 0.16, 1.0), (0, 0, -1), 0.5, (128,) * 3, 0, 0.5, 2.0, 0),
    "one": lambda: (np.array([[0.1, 0.1, 0.1]], np.float32), 0.05, (0.1, 0.1, 1.0), (0, 0, -1), 0.3, (128,) * 3, 0,
                    0.5, 2.0, 0),
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("mixed", [False, True])
def test_depth_equals_oracle(oracle_mod, name, mixed):
    from newton_sph_dev_b200.sensors import march_steps

    x, radius, pos, direction, fov, dims, sr, step, far, steps = CASES[name]()
    rng = np.random.default_rng(7)
    r = np.full(len(x), radius, np.float32)
    if mixed:  # radii over two decades, some absent, and outliers
        r *= (10 ** rng.uniform(-1.7, 0, len(x))).astype(np.float32)
        r[::29] = 0.0
        if len(x) > 100:
            x = x.copy()
            x[3], x[4], x[5] = (4e3, -2e3, 1e3), (-50.0, 7.0, 3.0), (3e7, 0.0, 0.0)
            r[6] = 20 * radius
    sr = float(np.float32(sr if sr else float(r.max()) + 1e-6))
    step = float(np.float32(step * sr))
    if not steps:
        steps = march_steps(far, step)[0]
    w, h = 44, 30
    cam, ocam = _camera(oracle_mod, pos, direction, (0.1, 1.0, 0.2), fov, w, h, far)
    init = np.full((h, w), np.float32(far), np.float32)
    init[::4, ::3] = rng.uniform(0.1, 1.2 * far, init[::4, ::3].shape).astype(np.float32)
    raw, _ = _device_depth(x, r, dims, cam, sr, step, steps, init)
    ref = oracle_mod.raycast_particles(x, r, dims, ocam, sr, step, steps, depth_init=init, clamp=False)
    np.testing.assert_array_equal(raw, ref)


@pytest.mark.parametrize("n", [2, 7, 8, 9, 63, 65, 513, 4097, 33000])
def test_tree_sizes(oracle_mod, n):
    """Node counts around the tree's arity, one level to five."""
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    r = np.full(n, np.float32(0.3 / n ** (1 / 3)), np.float32)
    sr = float(r[0]) + 1e-6
    cam, ocam = _camera(oracle_mod, (1.9, -0.8, 1.2), (-1.4, 1.3, -0.7), (0, 0, 1), 0.6, 40, 30, 4.0)
    step = 0.5 * sr
    steps = int(4.0 / step) + 1
    init = np.full((30, 40), np.float32(4.0), np.float32)
    raw, _ = _device_depth(x, r, (128, 128, 128), cam, sr, step, steps, init)
    ref = oracle_mod.raycast_particles(x, r, (128, 128, 128), ocam, sr, step, steps, depth_init=init, clamp=False)
    np.testing.assert_array_equal(raw, ref)


@pytest.mark.parametrize("offset", [0.0, 700.0, 2.0e5])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 24])
def test_few_hits(oracle_mod, k, offset):
    """Rays whose nearest hits no sample's box holds, and that cross as many
    spheres as the list of all hits has places, fewer and more; near the
    origin, and where coordinates are coarse."""
    rng = np.random.default_rng(k)
    column = np.zeros((k, 3), np.float32)
    column[:, 0] = np.linspace(0.0, 1.5, k)
    column[:, 1:] = rng.uniform(-0.03, 0.03, (k, 2))
    x = np.concatenate([column, rng.uniform(-0.5, 1.5, (200, 3))]).astype(np.float32) + np.float32(offset)
    r = np.full(len(x), 0.01, np.float32)
    r[:k] = rng.uniform(0.03, 0.2, k)  # much wider than the search radius
    far = 3.5
    pos = tuple(float(np.float32(offset) + np.float32(c)) for c in (-1.0, 0.003, -0.002))
    cam, ocam = _camera(oracle_mod, pos, (1, 0.001, 0.002), (0, 0, 1), 0.25, 36, 28, far)
    init = np.full((28, 36), np.float32(far), np.float32)
    for sr, step, dims in ((0.012, 0.006, (128,) * 3), (0.02, 0.013, (23, 16, 9)), (0.004, 0.0001, (64,) * 3)):
        sr, step = float(np.float32(sr)), float(np.float32(step))
        steps = int(far / step) + 2
        raw, _ = _device_depth(x, r, dims, cam, sr, step, steps, init)
        ref = oracle_mod.raycast_particles(x, r, dims, ocam, sr, step, steps, depth_init=init, clamp=False)
        np.testing.assert_array_equal(raw, ref)
