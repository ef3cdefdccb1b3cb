"""What reservations take, and that a step asks for no memory that its solver
could have had from the start."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def test_grid_reservation_stays_within_its_granules():
    """2^20 points: six sort buffers of 4 MiB, half a MiB of histograms and a
    mirror of 32 MiB, in granules of 2 MiB."""
    from newton_sph_dev_b200 import HashGrid

    HashGrid(16, 16, 16, device=DEV).reserve(1000)  # the kernels are loaded
    grid = HashGrid(16, 16, 16, device=DEV)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    grid.reserve(1 << 20)
    assert free - torch.cuda.mem_get_info()[0] <= 60 << 20
    grid.build(torch.rand((1 << 20, 3), device=DEV), 0.05)
    assert torch.equal(grid.point_ids.sort().values, torch.arange(1 << 20, dtype=torch.int32, device=DEV))


def test_first_xpbd_step_allocates_nothing():
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverXPBD

    n = 3000
    b = nsph.ModelBuilder()
    b.add_particles(pos=(np.random.default_rng(1).random((n, 3)) * 0.2).astype(np.float32),
                    vel=np.zeros((n, 3), np.float32), mass=np.full(n, 1.0), radius=np.full(n, 0.005))
    b.add_ground_plane()
    model = b.finalize(DEV)
    solver = SolverXPBD(model, iterations=3)
    s0, s1, contacts = model.state(), model.state(), model.contacts()
    model.collide(s0, contacts)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    solver.step(s0, s1, None, contacts, 1e-3)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == held
    assert torch.cuda.max_memory_allocated() == held


def test_segment_tape_takes_what_it_says():
    """372 bytes per particle and 8 per cell, per step (64 steps of 16,384
    particles on 16^3 cells: 8 bytes more each would be 8 MiB)."""
    import newton_sph_dev_b200 as nsph
    from newton_sph_dev_b200.solvers import SolverSPH

    n, steps = 16384, 64
    b = nsph.ModelBuilder()
    b.add_particles(pos=(np.random.default_rng(1).random((n, 3)) * 0.3).astype(np.float32),
                    vel=np.zeros((n, 3), np.float32), mass=np.full(n, 1e-3))
    model = b.finalize(DEV)
    solver = SolverSPH(model, SolverSPH.Config(smoothing_length=0.02, grid_dims=(16, 16, 16)))
    solver.enable_adjoint()
    solver.reserve_segment(1)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    solver.reserve_segment(steps)
    first = (372 * n + 8 * 16**3) + 48 * n  # the tape of one step, given back
    took = free - torch.cuda.mem_get_info()[0]
    assert took <= steps * (372 * n + 8 * 16**3) + 48 * n - first + (6 << 20)
