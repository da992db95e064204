"""GPU: QMDFF torsions whose atoms are in line.

Where i-j-k or j-k-l lie exactly on a line the plane normal is the zero vector:
the reference takes the angle of the product as it is (src/valijkl.f90) and
leaves its derivative out (src/dphidr.f90).  Also a normal of 1e-15, which it does not
normalise, and one of 1e-9, which it does.  Energy and gradient of the plain form
against the oracle at its bar (1e-12), the mixed form finite; the adjoint's
derivatives finite, and H w along the line, where the gradient is smooth, against
central differences of the oracle's gradient (step 1e-4: 1e-5)."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
R = 2.9  # bohr

# i, j, k, l of one torsion
SHAPES = {
    "ijk": [[0, 0, 0], [0, 0, R], [0, 0, 2 * R], [1.9, 0.4, 2.7 * R]],
    "jkl": [[1.9, 0.4, -0.7 * R], [0, 0, 0], [0, 0, R], [0, 0, 2 * R]],
    "all": [[0, 0, 0], [0, 0, R], [0, 0, 2 * R], [0, 0, 3 * R]],
    "on x, folded back": [[0, 0, 0], [R, 0, 0], [2 * R, 0, 0], [1.2 * R, 0, 0]],
    "normal of 1e-15": [[3e-16, 0, 0], [0, 0, R], [0, 0, 2 * R], [1.9, 0.4, 2.7 * R]],
    "normal of 1e-9": [[3e-10, 0, 0], [0, 0, R], [0, 0, 2 * R], [1.9, 0.4, 2.7 * R]],
}


def chain():
    ref = np.array([[0.0, 0.0, 0.0], [2.7, 0.8, 0.0], [4.6, -1.4, 0.3], [7.2, -0.5, 1.1]])
    return Q.from_topology([6, 6, 6, 1], ref, [(0, 1), (1, 2), (2, 3)])


@pytest.mark.parametrize("shape", list(SHAPES))
def test_torsion_in_line_matches_oracle(require_gpu, shape):
    ff, tab = chain(), Q.ElementTables.caracal()
    assert len(ff.tors) == 1
    orc.set_qmdff(ff, tab)
    g = QMDFFForceField(ff, tab)
    x = np.repeat(np.array(SHAPES[shape])[None], 3, axis=0)
    eo, go = orc.egrad("qmdff", x)
    assert np.isfinite(eo).all() and np.isfinite(go).all()
    e, grad = g.egrad(x, "fp64")
    assert np.isfinite(e).all() and np.isfinite(grad).all()
    assert rel_err(e, eo) <= 1e-12 and rel_err(grad, go) <= 1e-12
    em, gm = g.egrad(x, "mixed")
    assert np.isfinite(em).all() and np.isfinite(gm).all()
    # w leaves the line as it is: the gradient is smooth along it
    w = np.zeros_like(x)
    axis = 0 if "on x" in shape else 2
    w[:, :, axis] = np.array([0.3, -0.2, 0.5, 0.1])
    ev, gv, hw = g.hvp(x, w)
    assert rel_err(ev, eo) <= 1e-12 and rel_err(gv, go) <= 1e-12 and np.isfinite(hw).all()
    if shape in ("ijk", "jkl", "all"):
        h = 1e-4
        num = (orc.egrad("qmdff", x + h * w)[1] - orc.egrad("qmdff", x - h * w)[1]) / (2 * h)
        # truncation h^2 of the third derivatives over the second ones, rounding 1e-16 / h
        assert rel_err(hw, num) <= 1e-5
    v = np.random.default_rng(1).normal(size=x.shape)
    grads = g.param_vjp(x, v)
    assert np.isfinite(grads).all()
    g.close()
