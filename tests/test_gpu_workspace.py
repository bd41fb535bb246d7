"""A plan whose workspace could not grow for one run: the next run, of a shape
that fitted before, gets memory at the old address that no longer holds its box
table, and gives the oracle's catalog all the same."""
import pytest

import cm_halofinder_b200 as cmh
from cm_halofinder_b200 import FofConfig, Plan, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu

OOM = 4


@pytest.mark.parametrize("varlink", [False, True])
@pytest.mark.parametrize("graph", [True, False])
def test_run_after_one_that_did_not_fit(graph, varlink, monkeypatch):
    import torch
    n = 60_000
    if varlink:
        w = synth.make_lightcone(n, 1400.0 * (n / 50_000_000) ** (1 / 3), 150, 621)
    else:
        w = synth.config2(seed=621, scale=n / 256 ** 3)
    ref = cpu.run(w)
    pos, vel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    plan = Plan(FofConfig.from_workload(w))
    plan.set_graph(graph)
    try:
        for _ in range(2):
            for _ in range(2):
                assert_same_catalog(plan.run(pos, vel), ref, check_member=False)
            monkeypatch.setenv("CMH_FAULT", "alloc")
            with pytest.raises(cmh.CmhError) as e:   # (the membership needs more room)
                plan.run(pos, vel, members=True)
            assert e.value.status == OOM
            with pytest.raises(cmh.CmhError):
                plan.run(pos, vel)
            monkeypatch.delenv("CMH_FAULT")
            # other work may have been given the memory meanwhile
            other = torch.full((1 << 24,), 0x7f7f7f7f, dtype=torch.int32, device="cuda")
            del other
            torch.cuda.empty_cache()
        assert_same_catalog(plan.run(pos, vel), ref, check_member=False)
        for _ in range(2):
            assert_same_catalog(plan.run(pos, vel, members=True), ref)
    finally:
        plan.close()
