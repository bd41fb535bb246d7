"""Catalogs handed to the caller: the whole membership and the halo indices
alone through the C ABI, large memberships that stay the library's memory, and
records that pass through pinned memory from a plan's second run on."""
import ctypes as C
import gc

import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, Plan, _abi, fof, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("want", [1, -1, _abi.CMH_MEMBER_INDEX])
def test_membership_through_the_c_abi(want):
    w = synth.config2(seed=501, scale=20000 / 256 ** 3)
    ref = cpu.run(w)
    src, ppos, _ = cpu.build_proc(w)
    p = FofConfig.from_workload(w).to_c()
    parts = _abi.Particles(n=w.n, pos_dtype=0, vel_dtype=0, pos=w.pos.ctypes.data,
                           vel=w.vel.ctypes.data, id=None, location=_abi.CMH_HOST)
    cat = _abi.Catalog()
    L = _abi.lib()
    _abi.check(L.cmh_fof_run(C.byref(p), C.byref(parts), C.byref(cat), want, None))
    try:
        member = np.ctypeslib.as_array(cat.member, shape=(w.n,))
        np.testing.assert_array_equal(member, ref["member"])
        if want == _abi.CMH_MEMBER_INDEX:
            assert not cat.member_proc and not cat.member_pos
        else:
            ins = np.nonzero(member >= 0)[0]
            proc = np.ctypeslib.as_array(cat.member_proc, shape=(w.n,))[ins]
            np.testing.assert_array_equal(np.asarray(src)[proc], ins)
            got = np.ctypeslib.as_array(cat.member_pos, shape=(w.n, 3))[ins]
            np.testing.assert_array_equal(got, np.asarray(ppos)[proc])
    finally:
        L.cmh_catalog_free(C.byref(cat))


def test_large_membership_outlives_its_catalog():
    import torch
    w = synth.config2(seed=502, scale=150000 / 256 ** 3)
    ref = cpu.run(w)
    cfg = FofConfig.from_workload(w)
    member = fof(w.pos, w.vel, cfg, members=True).member
    plan = Plan(cfg)
    pos, vel = torch.from_numpy(w.pos).cuda(), torch.from_numpy(w.vel).cuda()
    cats = [plan.run(pos, vel, members=True) for _ in range(4)]
    plan.close()
    gc.collect()
    for cat in cats:
        assert_same_catalog(cat, ref)
    tail = cats.pop().member[-1000:]
    cats.clear()
    gc.collect()
    np.testing.assert_array_equal(member, ref["member"])
    np.testing.assert_array_equal(tail, ref["member"][-1000:])


@pytest.mark.parametrize("cells", [1, 31, 32, 33, 65])
def test_sizes_and_heads_by_cells(cells):
    """Group sizes are counted a fine cell at a time and heads found for the
    candidates alone: a chain of cells of one to three particles each and lone
    particles, every group a candidate (1 member), in shuffled input order."""
    rng = np.random.default_rng(cells)
    chain = np.repeat(np.arange(cells), 1 + np.arange(cells) % 3)
    pts = np.full((len(chain), 3), 5.0)
    pts[:, 0] = 2.0 + 0.045 * chain
    lone = np.stack([1.0 + 0.2 * np.arange(cells // 2), *np.full((2, cells // 2), 8.0)], 1)
    pos = rng.permutation(np.concatenate([pts, lone])).astype(np.float32)
    w = synth.Workload(name="chain", pos=pos, vel=rng.normal(0, 300, pos.shape).astype(np.float32),
                       ids=np.arange(len(pos), dtype=np.uint64), lo=(0.0,) * 3, hi=(10.0,) * 3,
                       linklength=0.05, boundary=1.0, nphalomin=1, periodic=False, cells=100)
    cat = fof(w.pos, w.vel, FofConfig.from_workload(w), members=True)
    assert cat.nhalos == 1 + cells // 2
    assert_same_catalog(cat, cpu.run(w))
