"""Smallest group sizes that are no ordinary number: not above 1, NaN (no count
is below it: every group is a halo) and infinity (none is)."""
import pytest

from cm_halofinder_b200 import FofConfig, Plan, fof, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [1.0, 0.5, 0.0, -3.0, float("nan"), float("-inf"), 1.5, float("inf")])
def test_unusual_cuts(cut):
    import torch
    w = synth.config2(seed=641, scale=20000 / 256 ** 3)
    w.nphalomin = 2 if cut == 1.5 else 1
    ref = cpu.run(w)
    cfg = FofConfig.from_workload(w)
    cfg.nphalomin = cut
    cat = fof(w.pos, w.vel, cfg, members=True)
    if cut == float("inf"):
        assert cat.nhalos == 0 and (cat.member == -1).all()
        return
    assert_same_catalog(cat, ref)
    # in a batch with a box of another cut
    w2 = synth.config2(seed=642, scale=10000 / 256 ** 3)
    pos = [torch.from_numpy(v.pos).cuda() for v in (w2, w)]
    vel = [torch.from_numpy(v.vel).cuda() for v in (w2, w)]
    cfgs = [FofConfig.from_workload(w2), cfg]
    plan = Plan(cfgs[0])
    for _ in range(2):
        a, b = plan.run_batch(cfgs, pos, vel)
        assert_same_catalog(a, cpu.run(w2), check_member=False)
        assert_same_catalog(b, ref, check_member=False)
    plan.close()
