"""Plans of different cell sizes run at the same time from several threads, each
on a stream of its own: the dense top cells' kernel needs another amount of shared
memory in each."""
import threading

import pytest

from cm_halofinder_b200 import FofConfig, Plan, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


def test_plans_of_different_cell_sizes_in_threads():
    import torch
    w = synth.config2(seed=661, scale=30000 / 256 ** 3)
    ref = cpu.run(w)
    errors = []

    def work(cell_factor):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                pos, vel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
            stream.synchronize()
            plan = Plan(FofConfig.from_workload(w, cell_factor=cell_factor))
            plan.set_graph(False)
            try:
                for _ in range(150):
                    assert_same_catalog(plan.run(pos, vel, stream=stream), ref,
                                        check_member=False)
            finally:
                plan.close()
        except Exception as e:
            errors.append((cell_factor, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in (4, 8, 20, 32)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
