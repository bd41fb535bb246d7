"""Groups whose fine cells hang in long chains of the union-find when the last
compression starts, run after run: every member counts, is summed and carries
its halo's index, against the oracle."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell_factor", [2, 4, 8])
def test_long_chains(cell_factor):
    """144 lines of 500 particles 0.95 l apart (mostly two fine cells apart, so
    that the last pass over the far pairs joins them), in dense top cells."""
    import torch
    rng = np.random.default_rng(cell_factor)
    m, l = 500, 1.0
    x, y, z = np.meshgrid(2.0 + 0.95 * np.arange(m), 2.0 + 2.2 * np.arange(12),
                          2.0 + 2.2 * np.arange(12), indexing="ij")
    pos = np.stack([x, y, z], -1).reshape(-1, 3)
    pos[:, 1:] += rng.uniform(-0.05, 0.05, (len(pos), 2))
    pos = np.ascontiguousarray(rng.permutation(pos)).astype(np.float32)
    L = float(pos.max()) + 2.0
    w = synth.Workload(name="lines", pos=pos, vel=rng.normal(0, 300, pos.shape).astype(np.float32),
                       ids=np.arange(len(pos), dtype=np.uint64), lo=(0.0,) * 3, hi=(L,) * 3,
                       linklength=l, boundary=1.0, nphalomin=2, periodic=False, cells=60)
    ref = cpu.run(w)
    assert (ref["halo_props"][:, 0] == m).all() and len(ref["halo_head"]) == 144
    plan = Plan(FofConfig.from_workload(w, cell_factor=cell_factor))
    plan.set_tuning({"cell_scale": 1.0, "dense_min": 1})
    dpos, dvel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    for _ in range(25):
        cat = plan.run(dpos, dvel, members=True)
        assert_same_catalog(cat, ref)
        assert cat.stats["n_groups"] == 144
    plan.close()
