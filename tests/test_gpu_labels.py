"""Allocation-free labels on inputs where the fine-cell path can go wrong,
against every pair tested with the reference's predicate: sizes around a warp
and a block, crowded cells, coincident particles, probes that wrap around the
hash table's end being as likely as any, and domains of so many fine cells
that the coarse grid is kept."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, synth
from tests.test_zz_no_alloc import _brute_labels, _labels_noalloc

pytestmark = pytest.mark.gpu


def config(L, l, b=0.0):
    return FofConfig(lo=(0.0,) * 3, hi=(L,) * 3, boundary=b, linklength=l, nphalomin=1,
                     periodic=False, precision="fp64")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 3000])
def test_sizes(n, dtype):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * 10.0).astype(dtype)
    l = 0.9 * 10.0 / max(n, 2) ** (1 / 3)
    np.testing.assert_array_equal(_labels_noalloc(pos, config(10.0, l)), _brute_labels(pos, l))


@pytest.mark.parametrize("crowd", [1, 5, 33, 200])
@pytest.mark.parametrize("inside", [True, False])
def test_one_pair_decides(crowd, inside):
    """Two crowds whose nearest particles are l (1 -+ 1e-4) apart, all others
    behind them, forty times over."""
    rng = np.random.default_rng(crowd)
    m, l = (40 if crowd < 100 else 8), 1.0
    c = rng.uniform(5.0, 395.0, (m, 1, 3))
    d = rng.standard_normal((m, 1, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    t = rng.uniform(0.0, 0.05, (m, crowd, 1))
    t[:, 0] = 0.0
    b = c + d * l * (1.0 - 1e-4 if inside else 1.0 + 1e-4) + t * d
    pos = rng.permutation(np.concatenate([(c - t * d).reshape(-1, 3), b.reshape(-1, 3)]))
    label = _labels_noalloc(np.ascontiguousarray(pos), config(400.0, l))
    np.testing.assert_array_equal(label, _brute_labels(pos, l))
    assert len(np.unique(label)) == (m if inside else 2 * m)


def test_full_table_and_one_cell():
    """65,536 particles: each alone in its cell, and all in one."""
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(n) for n in (64, 32, 32)], indexing="ij"), -1)
    pos = np.ascontiguousarray(rng.permutation(g.reshape(-1, 3) + 0.5)).astype(np.float32)
    np.testing.assert_array_equal(_labels_noalloc(pos, config(64.0, 0.9)), np.arange(65536))
    one = np.full((65536, 3), 7.25, np.float32) + rng.uniform(0, 0.01, (65536, 3)).astype(np.float32)
    assert not _labels_noalloc(one, config(64.0, 0.9)).any()


@pytest.mark.parametrize("l", [2e-3, 4e-4])
def test_huge_domain(l):
    """About 2^39.7 and 2^42 fine cells an axis: fine cells and coarse grid."""
    rng = np.random.default_rng(9)
    L = 1.0e9
    base = rng.random((300, 3)) * L
    near = base[:200] + rng.choice([-1.0, 1.0], (200, 3)) * (0.5 * l)
    far = base[200:] + rng.choice([-1.0, 1.0], (100, 3)) * (1.5 * l)
    pos = rng.permutation(np.clip(np.concatenate([base, near, far]), 0.0, L))
    label = _labels_noalloc(np.ascontiguousarray(pos), config(L, l))
    np.testing.assert_array_equal(label, _brute_labels(pos, l))
    assert len(np.unique(label)) < len(pos)


def test_benchmark_distribution_of_one_clump():
    w = synth.config2(seed=21, scale=6000 / 256 ** 3)
    cfg = FofConfig(lo=w.lo, hi=w.hi, boundary=0.0, linklength=w.linklength, nphalomin=1,
                    periodic=False, precision="fp64")
    np.testing.assert_array_equal(_labels_noalloc(w.pos, cfg), _brute_labels(w.pos, w.linklength))
