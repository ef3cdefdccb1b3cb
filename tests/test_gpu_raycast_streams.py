"""Raycasts of one grid from several streams and host threads: the calls share
the grid's work memory, so each waits for the one before, and every image is
the one that a call alone gives."""

from __future__ import annotations

import ctypes
import threading

import numpy as np
import pytest
import torch

from test_gpu_raycast import _camera

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("threads", [False, True])
def test_cameras_on_streams_of_their_own(oracle_mod, threads):
    from newton_sph_dev_b200 import HashGrid, _lib

    n, far, w, h = 30000, 4.0, 80, 60
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32)).to(DEV)
    r = torch.full((n,), 0.006, device=DEV)
    sr = float(np.float32(0.006 + 1e-6))
    grid = HashGrid(128, 128, 128, device=DEV)
    grid.reserve(n)
    grid.build(x, sr)
    views = [((1.9, -0.8, 1.2), (-1.4, 1.3, -0.7)), ((-0.9, 0.4, 0.3), (1.4, 0.1, 0.2)), ((0.5, 0.5, 0.5), (0.2, 0.3, 1.0))]
    cams = [_camera(oracle_mod, p, d, (0, 0, 1) if i < 2 else (0, 1, 0), 0.7 + 0.3 * i, w, h, far)[0]
            for i, (p, d) in enumerate(views)]
    lib = _lib.load()

    def shoot(cam, depth, stream):
        _lib.check(lib.nsph_raycast_particles(grid.id, x.data_ptr(), r.data_ptr(), n, ctypes.byref(cam), sr, 0.5 * sr,
                                              int(far / (0.5 * sr)) + 2, depth.data_ptr(),
                                              ctypes.c_void_p(stream.cuda_stream)), "raycast")

    alone = []
    for cam in cams:
        depth = torch.full((h, w), far, device=DEV)
        shoot(cam, depth, torch.cuda.current_stream())
        torch.cuda.synchronize()
        alone.append(depth)
    assert all((a < far).any() for a in alone) and not torch.equal(alone[0], alone[1])

    streams = [torch.cuda.Stream(DEV) for _ in cams]
    images = [[torch.full((h, w), far, device=DEV) for _ in range(12)] for _ in cams]
    torch.cuda.synchronize()

    def row(i):
        for depth in images[i]:
            shoot(cams[i], depth, streams[i])

    if threads:
        failed = []

        def guarded(i):
            try:
                row(i)
            except Exception as e:  # noqa: BLE001
                failed.append(e)

        workers = [threading.Thread(target=guarded, args=(i,)) for i in range(len(cams))]
        [t.start() for t in workers]
        [t.join() for t in workers]
        assert not failed
    else:
        for k in range(12):
            for i, s in enumerate(streams):
                shoot(cams[i], images[i][k], s)
    torch.cuda.synchronize()
    for a, row_ in zip(alone, images):
        assert all(torch.equal(a, b) for b in row_)
