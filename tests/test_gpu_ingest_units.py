"""Domain filter and periodic images of boxes in very large units (FP64
positions), against the oracle: a face, or the shell's inner edge, at 0 while the
box spans so many units that rounding at its far side is larger than 2."""
import numpy as np
import pytest

from cm_halofinder_b200 import FofConfig, fof, synth
from oracle import cpu
from tests.helpers import assert_same_catalog

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("edge", ["lo", "hi", "image_by_plus", "image_by_minus", "shell_lo",
                                  "shell_hi"])
@pytest.mark.parametrize("L", [3e16, 3e22])
def test_an_edge_at_zero(L, edge, periodic):
    """Particles at exactly 0, one value on either side of it, and up to a few
    times the far side's rounding around it; nothing is linked, so that every
    particle is its own halo."""
    b = 0.01 * L
    lo = {"lo": 0.0, "hi": -L, "image_by_plus": -b, "image_by_minus": b - L, "shell_lo": b,
          "shell_hi": -L - b}[edge]
    rng = np.random.default_rng(31)
    n, ulp = 1500, np.spacing(L)
    pos = lo + rng.random((n, 3)) * L
    near = np.concatenate([[0.0, 5e-324, 1.0], ulp * np.array([0.5, 1.0, 4.0, 9.0, 20.0])])
    near = np.concatenate([near, -near])
    some = np.nonzero(rng.random(n) < 0.6)[0]
    pos[some, rng.integers(0, 3, len(some))] = near[rng.integers(0, len(near), len(some))]
    w = synth.Workload(name="units", pos=pos, vel=rng.normal(0, 300, (n, 3)).astype(np.float32),
                       ids=np.arange(n, dtype=np.uint64), lo=(lo,) * 3, hi=(lo + L,) * 3,
                       linklength=0.002 * L / n ** (1 / 3), boundary=b, nphalomin=1,
                       periodic=periodic, cells=8)
    ref = cpu.run(w)
    cat = fof(w.pos, w.vel, FofConfig.from_workload(w, precision="fp64"), members=True)
    for count in ("n_out", "n_images"):
        assert cat.stats[count] == ref["stats"][count]
    assert_same_catalog(cat, ref)
