"""Domain filter, periodic images and processing order where the ingest can go
wrong, against the oracle: coordinates within a few representable values of
the faces and of the shell's inner edge, domains away from the origin and
around it, sizes around a tile and around a group of the catalog's heads,
unaligned device arrays, empty boxes in a
batch."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan, fof, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


def workload(lo, L, b, n, dtype, periodic, seed):
    """Random particles, each with one coordinate (for half of them) a few
    representable values around a face, an edge of the shell or its inner image.
    Nothing is linked, so every particle is its own halo and whether it is
    owned does not hang on the rounding of a sum."""
    rng = np.random.default_rng(seed)
    lo = np.asarray(lo, np.float64)
    pos = (lo + rng.random((n, 3)) * L).astype(dtype)
    axis = rng.integers(0, 3, n)
    edge = np.stack([lo, lo + L, lo + b, lo + L - b, lo - b, lo + L + b])
    x = edge[rng.integers(0, 6, n), axis].astype(dtype)
    for _ in range(3):
        x = np.where(rng.random(n) < 0.5, np.nextafter(x, dtype(np.inf)),
                     np.nextafter(x, dtype(-np.inf)))
    some = np.nonzero(rng.random(n) < 0.5)[0]
    pos[some, axis[some]] = x[some]
    vel = rng.normal(0, 300, (n, 3)).astype(np.float32)
    return synth.Workload(name="edges", pos=pos, vel=vel, ids=np.arange(n, dtype=np.uint64),
                          lo=tuple(lo), hi=tuple(lo + L), linklength=0.005 * L / n ** (1 / 3),
                          boundary=b, nphalomin=1, periodic=periodic,
                          cells=max(int(0.5 * n ** (1 / 3)), 1))


def check(w, cat, ref):
    assert_same_catalog(cat, ref)
    assert cat.stats["n_out"] == ref["stats"]["n_out"]


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("lo,L,b", [((0.0, 0.0, 0.0), 100.0, 7.0), ((-7.0, -50.0, 41.3), 100.0, 7.0),
                                    ((-93.0, 1000.7, -1e4), 100.0, 7.0),
                                    ((0.0, 0.0, 0.0), 10.0, 6.0)])
def test_faces_and_shell_edges(lo, L, b, dtype, periodic):
    w = workload(lo, L, b, 3000, dtype, periodic, 3)
    check(w, fof(w.pos, w.vel, FofConfig.from_workload(w), members=True), cpu.run(w))


@pytest.mark.parametrize("n", [3, 4, 5, 1023, 1024, 1025, 4097])
def test_sizes_and_unaligned_arrays(n):
    import torch
    w = workload((0.0,) * 3, 50.0, 4.0, n, np.float32, True, n)
    ref = cpu.run(w)
    plan = Plan(FofConfig.from_workload(w))
    vel = torch.from_numpy(w.vel).cuda()
    for shift in (0, 1, 2, 3):
        room = torch.zeros(3 * n + shift, dtype=torch.float32, device="cuda")
        pos = room[shift:].view(n, 3)
        pos.copy_(torch.from_numpy(w.pos))
        check(w, plan.run(pos, vel, members=True), ref)
    plan.close()


def test_empty_boxes_in_a_batch():
    import torch
    ns = [0, 1500, 0, 0, 1, 1024, 2047, 0]
    ws = [workload((0.0,) * 3, 50.0, 4.0, max(n, 1), np.float32, True, 7 + i)
          for i, n in enumerate(ns)]
    pos = [torch.from_numpy(w.pos[:n]).cuda() for w, n in zip(ws, ns)]
    vel = [torch.from_numpy(w.vel[:n]).cuda() for w, n in zip(ws, ns)]
    cfgs = [FofConfig.from_workload(w) for w in ws]
    plan = Plan(cfgs[0])
    for _ in range(2):
        for w, n, cat in zip(ws, ns, plan.run_batch(cfgs, pos, vel)):
            if n == 0:
                assert cat.nhalos == 0
            else:
                assert_same_catalog(cat, cpu.run(w), check_member=False)
    plan.close()
