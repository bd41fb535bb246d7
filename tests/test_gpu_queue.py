"""More (fine cell, dense top cell) items than 32 bits count: each past the
queue's room is read cell by cell, and none takes an early item's place."""
import gc

import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan

pytestmark = pytest.mark.gpu


def test_items_beyond_32_bits():
    """A lattice of one particle per fine cell and eight per top cell: every
    forward neighbour of every cell is in reach, 13 items each where the
    neighbours have slots (a second run has slots for nearly half)."""
    import torch
    side, h = 950, 0.5
    if torch.cuda.mem_get_info()[0] < 150e9:
        pytest.skip("needs 150 GB of device memory")
    n = side ** 3
    g = h * (torch.arange(side, device="cuda", dtype=torch.float32) + 0.5)
    pos = torch.empty((side, side, side, 3), dtype=torch.float32, device="cuda")
    pos[..., 0] = g
    pos[..., 1] = g[:, None]
    pos[..., 2] = g[:, None, None]
    vel = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
    cfg = FofConfig(lo=(0.0,) * 3, hi=(side * h,) * 3, boundary=0.0,
                    linklength=h * np.sqrt(3.0) / (1.0 - 2.0 ** -20), nphalomin=1000,
                    periodic=False, cell_factor=2)
    plan = Plan(cfg)
    plan.set_tuning({"cell_scale": 1.0, "dense_min": 1})
    try:
        plan.run(pos.view(n, 3), vel)
        cat = plan.run(pos.view(n, 3), vel)
        assert cat.stats["n_cells"] == n and cat.stats["n_queued"] > 2 ** 32
        assert cat.nhalos == 1 and cat.stats["n_groups"] == 1
        assert cat.props[0, 0] == np.float32(n) and cat.head[0] == 0
        np.testing.assert_allclose(cat.props[0, 1:4], 0.5 * side * h, rtol=1e-6)
    finally:
        plan.close()
        del pos, vel
        gc.collect()
        torch.cuda.empty_cache()
