"""The ingest's tiles of 1024 particles (four per thread, read 16 bytes at a time
where the array's alignment allows) and the gather's large tiles, against the
oracle: runs just below and from the size where they begin, every remainder of a
thread's four and of a tile, unaligned arrays, and FP64 positions in several
buckets."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan, synth
from oracle import cpu
from tests.helpers import assert_same_catalog
from tests.test_gpu_ingest import check, workload

pytestmark = pytest.mark.gpu

FOUR = 148 * 4 * 256 * 4     # particles from which a thread takes four


@pytest.mark.parametrize("dtype,shifts", [(np.float32, (0, 1, 2, 3)), (np.float64, (0, 1))])
@pytest.mark.parametrize("n", [FOUR - 1, FOUR, FOUR + 1, FOUR + 2, FOUR + 3, FOUR + 1023])
def test_four_per_thread_and_unaligned_arrays(n, dtype, shifts):
    import torch
    w = workload((0.0,) * 3, 400.0, 4.0, n, dtype, True, n % 1000)
    ref = cpu.run(w)
    plan = Plan(FofConfig.from_workload(w), pos_dtype=dtype)
    vel = torch.from_numpy(w.vel).cuda()
    src = torch.from_numpy(w.pos).cuda()
    for shift in shifts:
        room = torch.zeros(3 * n + shift, dtype=src.dtype, device="cuda")
        pos = room[shift:].view(n, 3)
        pos.copy_(src)
        check(w, plan.run(pos, vel, members=True), ref)
    plan.close()


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_large_box_of_double_positions(precision):
    """2.9M FP64 particles: three buckets, the 2048-element gather."""
    import torch
    w = synth.make_box(2_900_003, 560.0, 1700, 651, pos_dtype=np.float64)
    ref = _ref(w)
    plan = Plan(FofConfig.from_workload(w, precision=precision), pos_dtype=np.float64)
    pos, vel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    for _ in range(2):
        assert_same_catalog(plan.run(pos, vel, members=True), ref)
    plan.close()


_refs = {}


def _ref(w):
    if w.n not in _refs:
        _refs[w.n] = cpu.run(w)
    return _refs[w.n]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_batch_of_uneven_boxes_above_the_size(dtype):
    """Boxes of other sizes than whole tiles, empty ones among them, in one run of
    four particles per thread."""
    import torch
    ns = [300_001, 0, 1, 1023, 200_002, 0, 150_007]
    ws = [workload((0.0,) * 3, 50.0 + 5 * i, 4.0, max(n, 1), dtype, True, 40 + i)
          for i, n in enumerate(ns)]
    assert sum(ns) >= FOUR
    pos = [torch.from_numpy(w.pos[:n]).cuda() for w, n in zip(ws, ns)]
    vel = [torch.from_numpy(w.vel[:n]).cuda() for w, n in zip(ws, ns)]
    cfgs = [FofConfig.from_workload(w) for w in ws]
    plan = Plan(cfgs[0], pos_dtype=dtype)
    for _ in range(2):
        for w, n, cat in zip(ws, ns, plan.run_batch(cfgs, pos, vel)):
            if n == 0:
                assert cat.nhalos == 0
            else:
                assert_same_catalog(cat, cpu.run(w), check_member=False)
    plan.close()
