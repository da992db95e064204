"""GPU: Hessian-vector products of small and larger molecules.

A bead's block has as many warps as the largest kind of terms fills, one to eight: the
product against central differences of the oracle's gradient (step 1e-4: truncation and
rounding 1e-5 at most), the energy and gradient that come with it at the plain form's bar,
and a bead of a batch as the bead alone, bit for bit."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [2, 3, 4, 6, 10, 20])
def test_hvp(require_gpu, nc):
    ff, tab = Q.alkane(nc=nc), Q.ElementTables.caracal()
    orc.set_qmdff(ff, tab)
    g = QMDFFForceField(ff, tab)
    rng = np.random.default_rng(nc)
    x = ff.xyz[None] + rng.normal(0, 0.05, (613,) + ff.xyz.shape)
    w = rng.normal(0, 1, x.shape)
    e, grad, hw = g.hvp(x, w)
    few = slice(0, 3)
    eo, go = orc.egrad("qmdff", x[few])
    assert rel_err(e[few], eo) <= 1e-12 and rel_err(grad[few], go) <= 1e-12
    h = 1e-4
    num = (orc.egrad("qmdff", x[few] + h * w[few])[1] - orc.egrad("qmdff", x[few] - h * w[few])[1]) / (2 * h)
    assert rel_err(hw[few], num) <= 1e-5
    for b in (0, 300, 612):
        one = g.hvp(x[b:b + 1], w[b:b + 1])
        assert all(np.array_equal(u[0], v[b]) for u, v in zip(one, (e, grad, hw)))
    g.close()
