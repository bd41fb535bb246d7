"""Bounded device waits that run out on a tile that publishes nothing
(CMH_FAULT), in every kernel that looks back: the run reports the timeout, and the
plan's next runs give the catalog of before.  No GPU fault, and no wait longer than
its few polls."""
import pytest

import cm_halofinder_b200 as cmh
from cm_halofinder_b200 import FofConfig, Plan, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu

TIMEOUT = 7


@pytest.mark.parametrize("n", [60_000, 1_400_000])   # tiles of 1024 and of 2048 elements
@pytest.mark.parametrize("kind,who", [("gather", "run count"), ("lookback", "radix sort"),
                                      ("lookback,gather", "radix sort")])
def test_wait_runs_out_then_recovery(n, kind, who, monkeypatch):
    import torch
    w = synth.config2(seed=611, scale=n / 256 ** 3)
    ref = cpu.run(w)
    pos, vel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    plan = Plan(FofConfig.from_workload(w))
    try:
        for graph in (True, False):
            plan.set_graph(graph)
            assert_same_catalog(plan.run(pos, vel, members=True), ref)
            plan.set_limits(lookback_polls=20000)   # (some 10 ms: no other wait runs out)
            monkeypatch.setenv("CMH_FAULT", kind)
            for _ in range(2):
                with pytest.raises(cmh.CmhError) as e:
                    plan.run(pos, vel, members=True)
                assert e.value.status == TIMEOUT and f"{who} look-back" in str(e.value)
            monkeypatch.delenv("CMH_FAULT")
            plan.set_limits()
        # no poll at all: whichever wait comes first, if any
        plan.set_limits(lookback_polls=0)
        for _ in range(3):
            try:
                assert_same_catalog(plan.run(pos, vel, members=True), ref)
            except cmh.CmhError as e:
                assert e.status == TIMEOUT and "look-back" in str(e)
        plan.set_limits()
        for _ in range(2):
            assert_same_catalog(plan.run(pos, vel, members=True), ref)
    finally:
        plan.close()
