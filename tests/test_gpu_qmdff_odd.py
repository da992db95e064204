"""GPU: mixed QMDFF forces of molecules with an odd number of atoms.

Every warp of a block holds one bead in its own shared memory; with an odd atom
count the regions must not share a word, so a batch gives each bead exactly
what a call on that bead alone gives, and every repetition the same."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [3, 5, 7])
def test_batch_equals_single_beads(require_gpu, nc):
    ff = Q.alkane(nc=nc)
    assert ff.n % 2 == 1
    g = QMDFFForceField(ff)
    x = ff.xyz + np.random.default_rng(5).normal(0, 0.1, (1500,) + ff.xyz.shape)
    e, f = g.egrad(x, "mixed")
    for _ in range(20):
        e2, f2 = g.egrad(x, "mixed")
        assert np.array_equal(e2, e) and np.array_equal(f2, f)
    for b in range(0, 1500, 97):
        e1, f1 = g.egrad(x[b], "mixed")
        assert np.array_equal(e1[0], e[b]) and np.array_equal(f1[0], f[b])
    g.close()
