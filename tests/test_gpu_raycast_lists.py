"""Rays that cross as many spheres as the list of a ray's hits has places (32),
one fewer, one more and many more, none of whose nearest hits a sample's box
holds: the full list, and past it the march over windows of the grid's cells,
against the oracle's full march, near the origin (cells of known place) and
with grids that alias."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_raycast import _camera, _device_depth

pytestmark = pytest.mark.gpu


def _directions(cam):
    px, py = np.meshgrid(np.arange(cam.width), np.arange(cam.height))
    cx = ((2 * px + 1) / cam.width - 1) * cam.fov_scale * cam.aspect_ratio
    cy = (1 - (2 * py + 1) / cam.height) * cam.fov_scale
    d = cx[..., None] * np.array(cam.right[:]) + cy[..., None] * np.array(cam.up[:]) + np.array(cam.direction[:])
    return d / np.linalg.norm(d, axis=-1, keepdims=True)


@pytest.mark.parametrize("k", [31, 32, 33, 70])
@pytest.mark.parametrize("sr,step,dims", [(0.012, 0.006, (128,) * 3), (0.02, 0.013, (23, 16, 9)),
                                          (0.004, 0.0001, (64,) * 3)])
def test_list_boundary(oracle_mod, k, sr, step, dims):
    rng = np.random.default_rng(k)
    column = np.zeros((k, 3), np.float32)
    column[:, 0] = np.linspace(0.0, 0.08, k)  # their first hits lie within the first window
    column[:, 1:] = rng.uniform(-0.02, 0.02, (k, 2))
    x = np.concatenate([column, rng.uniform(-0.5, 1.5, (200, 3))]).astype(np.float32)
    r = np.full(len(x), 0.01, np.float32)
    r[:k] = rng.uniform(0.1, 0.2, k)  # much wider than the search radius, crossed by every ray near the axis
    far = 3.5
    cam, ocam = _camera(oracle_mod, (-1.0, 0.003, -0.002), (1, 0.001, 0.002), (0, 0, 1), 0.25, 36, 28, far)
    init = np.full((28, 36), np.float32(far), np.float32)
    sr, step = float(np.float32(sr)), float(np.float32(step))
    steps = int(far / step) + 2
    raw, _ = _device_depth(x, r, dims, cam, sr, step, steps, init)
    ref = oracle_mod.raycast_particles(x, r, dims, ocam, sr, step, steps, depth_init=init, clamp=False)
    np.testing.assert_array_equal(raw, ref)
    # many rays cross all of the column, and few of them end at their nearest hit
    d = _directions(cam)
    oc = np.array([-1.0, 0.003, -0.002]) - x.astype(np.float64)
    proj = d @ oc.T
    disc = proj * proj - ((oc * oc).sum(1) - r.astype(np.float64) ** 2)
    first = np.where(disc > 0, -proj - np.sqrt(np.maximum(disc, 0)), np.inf)
    all_of_them = (disc[..., :k] > 0).all(-1)
    later = ref > first.min(-1) + 1e-3
    assert all_of_them.sum() > 50
    if dims[0] > 23:  # (the small grid's early samples see the column's cells through their images)
        assert (all_of_them & later).sum() > 25
