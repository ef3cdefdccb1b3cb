"""The raycast where coordinates are coarse: camera and spheres far from the
origin, radii of a few last places of a coordinate down to a fraction of one.
The boxes of the tree have to hold every sphere that the march's own test hits,
so the depths are the oracle's full march's, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_raycast import _camera, _device_depth

pytestmark = pytest.mark.gpu


def _equal(oracle_mod, x, r, pos, direction, fov, sr, step, far, steps, w=56, h=40, dims=(128,) * 3):
    cam, ocam = _camera(oracle_mod, pos, direction, (0, 0, 1), fov, w, h, far)
    init = np.full((h, w), np.float32(far), np.float32)
    sr, step = float(np.float32(sr)), float(np.float32(step))
    raw, _ = _device_depth(x, r, dims, cam, sr, step, steps, init)
    ref = oracle_mod.raycast_particles(x, r, dims, ocam, sr, step, steps, depth_init=init, clamp=False)
    np.testing.assert_array_equal(raw, ref)
    return ref < np.float32(far)


@pytest.mark.parametrize("offset", [5e3, 1e4, 2e5])
@pytest.mark.parametrize("places", [0.3, 0.7, 1.0, 1.41, 1.5, 3.0, 4.2, 5.43, 6.0])
def test_boxes_hold_their_spheres(oracle_mod, offset, places):
    """A few spheres apart from one another (each on a face of its leaf's box),
    with more of them behind, radii in last places of the offset."""
    unit = float(np.spacing(np.float32(offset)))
    radius = np.float32(places * unit)
    rng = np.random.default_rng(int(offset) + int(100 * places))
    distance = 96 * max(1.0, places) * unit
    k = np.arange(-2, 3)
    side = distance / 6
    front = np.stack(np.meshgrid([0.0], k * side, k * side, indexing="ij"), -1).reshape(-1, 3)
    behind = front * 1.3 + [distance / 2, 0, 0]
    x = np.concatenate([front, behind]) + rng.uniform(-0.2, 0.2, (50, 3)) * side
    x = (x + offset).astype(np.float32)
    r = np.full(len(x), radius, np.float32)
    far = 3 * distance
    pos = tuple(float(np.float32(offset + c)) for c in (-distance, 0.0, 0.0))
    sr = max(float(radius) + 1e-6, 2 * unit)
    hits = 0
    # the whole sheet, and closer looks at parts of it
    for fov, dy, dz in ((0.8, 0.0, 0.0), (0.1, 0.0, 0.0), (0.1, 1.0, 0.0), (0.1, -1.0, 1.0), (0.1, 2.0, -2.0)):
        direction = (1.0, dy * side / distance, dz * side / distance)
        hits += _equal(oracle_mod, x, r, pos, direction, fov, sr, 0.5 * sr, far, int(far / (0.5 * sr)) + 2).sum()
    assert hits > 20


@pytest.mark.parametrize("offset", [5e3, 1e4, 2e5])
def test_block_far_from_the_origin(oracle_mod, offset):
    """A block of spheres of very different radii, many to a leaf."""
    unit = float(np.spacing(np.float32(offset)))
    rng = np.random.default_rng(3)
    size = 100 * unit
    x = (rng.uniform(0, size, (700, 3)) + offset).astype(np.float32)
    r = (unit * 10 ** rng.uniform(-0.5, 0.8, len(x))).astype(np.float32)
    pos = tuple(float(np.float32(offset + c * size)) for c in (-0.6, 0.4, 0.7))
    sr = float(r.max()) * 1.01
    far = 3 * size
    hits = _equal(oracle_mod, x, r, pos, (1.1, 0.1, -0.2), 0.9, sr, 0.4 * sr, far, int(far / (0.4 * sr)) + 2)
    assert hits.sum() > 100 and not hits.all()


@pytest.mark.parametrize("power", [62, 40, -40, -62, -70])
@pytest.mark.parametrize("name", ["inside", "overlap", "long_step", "truncated", "axis", "one"])
def test_scales(oracle_mod, name, power):
    """The same scenes in units in which distances are 10^18 and more, or their
    squares are denormal."""
    from newton_sph_dev_b200.sensors import march_steps
    from test_gpu_raycast_tree import CASES

    x, radius, pos, direction, fov, dims, sr, step, far, steps = CASES[name]()
    scale = 2.0**power
    sr = 1.0001 * radius
    if not steps:
        steps = march_steps(far, step * sr)[0]
    x = (x.astype(np.float64) * scale).astype(np.float32)
    r = np.full(len(x), radius * scale, np.float32)
    hits = _equal(oracle_mod, x, r, tuple(c * scale for c in pos), direction, fov, sr * scale, step * sr * scale,
                  far * scale, steps, dims=dims)
    assert hits.any()
