"""GPU: the plain QMDFF form by four warps per bead.

Molecules with fewer term batches than warps up to C20H42, batches of one bead
to more than the GPU holds at once: against the oracle at the plain form's bar
(1e-12), and every bead of a batch as the bead alone, bit for bit.  The
Hessian-vector product against central differences of the gradient (step 1e-4:
truncation about 1e-8 of the third derivative, rounding 1e-16 / 1e-4)."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,nbeads", [(3, 1), (3, 700), (6, 5), (13, 33), (20, 305)])
def test_team_matches_oracle(require_gpu, nc, nbeads):
    ff, tab = Q.alkane(nc=nc), Q.ElementTables.caracal()
    orc.set_qmdff(ff, tab)
    gff = QMDFFForceField(ff, tab)
    x = ff.xyz[None] + np.random.default_rng(nc).normal(0, 0.05, (nbeads,) + ff.xyz.shape)
    e, g = gff.egrad(x, "fp64")
    eo, go = orc.egrad("qmdff", x)
    assert rel_err(e, eo) <= 1e-12 and rel_err(g, go) <= 1e-12
    for b in (0, nbeads // 2, nbeads - 1):
        e1, g1 = gff.egrad(x[b:b + 1], "fp64")
        assert e1[0] == e[b] and np.array_equal(g1[0], g[b])
    gff.close()


def test_team_hvp(require_gpu):
    ff = Q.alkane(nc=4)
    gff = QMDFFForceField(ff)
    rng = np.random.default_rng(2)
    x = ff.xyz[None] + rng.normal(0, 0.05, (9,) + ff.xyz.shape)
    w = rng.normal(0, 1, x.shape)
    hw = gff.hvp(x, w)[-1]
    h = 1e-4
    num = (gff.egrad(x + h * w, "fp64")[1] - gff.egrad(x - h * w, "fp64")[1]) / (2 * h)
    assert rel_err(hw, num) <= 1e-5
    gff.close()
