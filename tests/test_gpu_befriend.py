"""Cell pairs that are hard to settle, against the oracle: crowded fine cells
whose one deciding particle pair is just inside or just outside the linking
length (one lane's bounded search, then the whole warp's), in sparse top
cells, in dense ones and across their faces (fine cells per top-cell edge from
the smallest to the largest), with few and with many queued cells."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan, fof, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


def crowded_pairs(crowd, inside, npairs, dtype, seed):
    """npairs pairs of crowds of `crowd` particles; the two nearest particles
    of a pair are l (1 -+ 1e-4) apart and the others lie behind them, so that
    pair alone decides.  A lattice of lone particles 1.3 l apart lies between,
    so that top cells of many fine cells are dense."""
    rng = np.random.default_rng(seed)
    L, l = 40.0, 1.0
    g = np.arange(0.65, L, 1.3 * l)
    lone = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    lone = lone + rng.uniform(-0.1, 0.1, lone.shape)
    c = rng.uniform(3.0, L - 3.0, (npairs, 1, 3))
    d = rng.standard_normal((npairs, 1, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    t = rng.uniform(0.0, 0.05, (npairs, crowd, 1))
    t[:, 0] = 0.0
    a = c - t * d
    b = c + d * l * (1.0 - 1e-4 if inside else 1.0 + 1e-4) + t * d
    keep = np.ones(len(lone), bool)
    for i in range(npairs):    # no lone particle near a pair
        keep &= np.linalg.norm(lone - c[i], axis=1) > 2.6 * l
    pos = np.concatenate([a.reshape(-1, 3), b.reshape(-1, 3), lone[keep]])
    pos = np.ascontiguousarray(rng.permutation(pos)).astype(dtype)
    return synth.Workload(name="crowds", pos=pos, vel=np.zeros(pos.shape, np.float32),
                          ids=np.arange(len(pos), dtype=np.uint64), lo=(0.0,) * 3, hi=(L,) * 3,
                          linklength=l, boundary=2.0, nphalomin=2, periodic=True, cells=20)


@pytest.mark.parametrize("inside", [True, False])
@pytest.mark.parametrize("crowd,npairs", [(1, 30), (6, 30), (33, 30), (200, 8)])
@pytest.mark.parametrize("cell_factor", [0, 4, 16, 32])
def test_one_pair_decides(cell_factor, crowd, npairs, inside):
    w = crowded_pairs(crowd, inside, npairs, np.float32, 17 * crowd + cell_factor)
    ref = cpu.run(w)
    for precision in ("fp32", "fp64"):
        cfg = FofConfig.from_workload(w, precision=precision, cell_factor=cell_factor)
        assert_same_catalog(fof(w.pos, w.vel, cfg, members=True), ref)


@pytest.mark.parametrize("cell_factor", [0, 32])
def test_one_pair_decides_double_positions(cell_factor):
    w = crowded_pairs(70, True, 10, np.float64, 5)
    cfg = FofConfig.from_workload(w, cell_factor=cell_factor)
    assert_same_catalog(fof(w.pos, w.vel, cfg, members=True), cpu.run(w))


@pytest.mark.parametrize("ratio", [1.0, 3.0, 9.0])
def test_reach_of_a_variable_length(ratio):
    """Windows of 5, 11 and 33 fine cells an axis (more than one word of rows)."""
    n = 30000
    w = synth.make_lightcone(n, 1400.0 * (n / 50_000_000) ** (1 / 3), 150, 61)
    tab = np.linspace(w.linklength / ratio, w.linklength, 65)
    w.varlink = {"origin": (0.0,) * 3, "rmax": float(w.hi[0]), "table": tab}
    assert_same_catalog(fof(w.pos, w.vel, FofConfig.from_workload(w), members=True), cpu.run(w))


@pytest.mark.parametrize("cell_factor,dense_min", [(4, 4), (8, 16), (3, 1)])
def test_queue_beyond_its_room(cell_factor, dense_min):
    """Near the percolation density with nearly every top cell dense and (but
    for the second case) every neighbour in reach: more (fine cell, dense top
    cell) pairs than the queue holds; those beyond are read cell by cell."""
    import torch
    rng = np.random.default_rng(71)
    n, l = 40000, 1.0
    L = (n / 0.6) ** (1 / 3)
    pos = (rng.random((n, 3)) * L).astype(np.float32)
    w = synth.Workload(name="uniform", pos=pos, vel=np.zeros_like(pos),
                       ids=np.arange(n, dtype=np.uint64), lo=(0.0,) * 3, hi=(L,) * 3,
                       linklength=l, boundary=2.0, nphalomin=5, periodic=False,
                       cells=int(L / 2))
    ref = cpu.run(w)
    plan = Plan(FofConfig.from_workload(w, cell_factor=cell_factor))
    plan.set_tuning({"cell_scale": 1.0, "dense_min": dense_min})
    dpos, dvel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    for _ in range(2):
        cat = plan.run(dpos, dvel, members=True)
        assert_same_catalog(cat, ref)
    if cell_factor != 8:
        assert cat.stats["n_queued"] > cat.stats["n_proc"]
    plan.close()
