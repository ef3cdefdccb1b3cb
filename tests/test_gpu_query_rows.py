"""The batched query's lanes-per-query form, bit-exact against the oracle's
candidate sequences where it can go wrong: one query and ragged counts, boxes
that wrap, boxes as wide as the grid, more rows than the lanes take, and
queries outside the 2^20 origin."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("dims,radius,qradius,nq,lo", [
    ((32, 32, 32), 0.05, 0.05, 1, 0.0), ((32, 32, 32), 0.05, 0.05, 33, 0.0), ((20, 17, 9), 0.03, 0.03, 200, -0.3),
    ((7, 5, 6), 0.05, 0.05, 100, 0.0), ((2, 2, 2), 0.05, 0.05, 50, 0.0), ((32, 32, 32), 0.05, 0.09, 100, 0.0),
    ((32, 32, 32), 0.05, 0.2, 60, 0.0), ((64, 64, 64), 0.02, 0.005, 100, 0.2), ((32, 32, 32), 0.05, 0.05, 40, -60000.0)])
def test_rows_equal_oracle(oracle_mod, dims, radius, qradius, nq, lo):
    from newton_sph_dev_b200 import HashGrid

    rng = np.random.default_rng(nq)
    pts = (rng.random((3000, 3)) * 0.7 + max(lo, -0.3)).astype(np.float32)
    q = (rng.random((nq, 3)) * 0.9 + lo).astype(np.float32)
    grid = HashGrid(*dims, device=DEV)
    grid.build(torch.from_numpy(pts).to(DEV), radius)
    offsets, ids = grid.query(torch.from_numpy(q).to(DEV), qradius)
    offsets, ids = offsets.cpu().numpy(), ids.cpu().numpy()
    ref = oracle_mod.grid_build(pts, radius, dims)
    inv = np.float32(1.0) / np.float32(radius)
    for t in range(nq):
        expect = oracle_mod.grid_query(ref, dims, inv, q[t], qradius)
        np.testing.assert_array_equal(ids[offsets[t]:offsets[t + 1]], expect, err_msg=f"query {t}")
