"""GPU: periodic boxes whose half edge is just below or above a bead's length.

Along a dimension in which a bead is shorter than half the edge the force
kernel skips the minimum image, elsewhere it takes it; the box edges here put
the line between the beads of a batch, below and above all of them.  Energies and
gradients against the oracle at the bars of the periodic tests (1e-12, 1e-11; the
edges stay far from the bonded vectors, whose dihedrals the reference takes from
raw coordinates); the mixed form within its stated error of the plain one."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField
from caracal_gb300 import qmdff as Q
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
BOHR = 0.52917721092


@pytest.mark.parametrize("factor", [1.98, 2.0, 2.003, 2.6])
def test_box_around_the_molecule(require_gpu, factor):
    ff, tab = Q.alkane(nc=6), Q.ElementTables.caracal()
    orc.set_qmdff(ff, tab)
    gff = QMDFFForceField(ff, tab)
    x = ff.xyz[None] + np.random.default_rng(8).normal(0, 0.05, (24,) + ff.xyz.shape)
    x[::2] = x[::2] - 40.0  # away from the origin
    extent = (x.max(1) - x.min(1)).mean(0)
    box = factor * extent * BOHR
    orc.set_qmdff_periodic(box, 50.0, 6.0)
    gff.set_periodic(box, 50.0, 6.0)
    e, g = gff.egrad(x, "fp64")
    eo, go = orc.egrad("qmdff", x)
    em, gm = gff.egrad(x, "mixed")
    gff.close()
    assert rel_err(e, eo) <= 1e-12 and rel_err(g, go) <= 1e-11
    assert np.sqrt(np.sum((gm - g) ** 2) / np.sum(g ** 2)) <= 1e-6
