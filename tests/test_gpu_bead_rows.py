"""GPU: the force kernels of a step evaluate one bead of each reflection pair.

After a drift in Caracal's modes beads j and P - j hold the same positions, so
the gradient row of every bead must equal a direct evaluation of its position,
bit for bit, for every bead count (none, one or several pairs, odd and even)."""
import numpy as np
import pytest

from caracal_gb300 import QMDFFForceField, RPMDEngine, WaterBox, egrad_h3
from caracal_gb300 import qmdff as Q
from caracal_gb300.units import beta_from_kelvin, dt_fs_to_au, mass_au
from caracal_gb300.water import water_box
from caracal_gb300.workloads import h3_collinear

pytestmark = pytest.mark.gpu


def stepped(pes, mass, q0, nbeads, ntraj, nm_mode, **kw):
    e = RPMDEngine(pes, mass, nbeads, ntraj, dt_fs_to_au(0.2), beta=beta_from_kelvin(300.0), seed=9,
                   nm_mode=nm_mode, **kw)
    e.init_positions(q0, 0.05)
    e.init_momenta()
    e.compute_forces()
    return e


@pytest.mark.parametrize("nbeads", [1, 2, 3, 5, 8, 24])
@pytest.mark.parametrize("nm_mode", [0, 1])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_qmdff_rows(require_gpu, nbeads, nm_mode, precision):
    ff = Q.alkane(nc=3)
    mass = [mass_au("C" if z == 6 else "H") for z in ff.at]
    g = QMDFFForceField(ff)
    e = stepped(g, mass, ff.xyz, nbeads, 3, nm_mode, thermostat="andersen", andersen_step=2, precision=precision)
    e.run(2)
    q, _, f, epot, st = e.get_state()
    V, want = g.egrad(q.reshape(-1, ff.n, 3), precision)
    assert not st.any() and np.array_equal(f.reshape(want.shape), want)
    assert np.allclose(epot, V.reshape(3, nbeads).sum(1), rtol=1e-13)
    e.close()


@pytest.mark.parametrize("nbeads", [2, 5, 8])
def test_umbrella_and_water_rows(require_gpu, nbeads):
    mech = dict(reac1=[1, 2], reac2=[3], bond_form=(2, 3), bond_break=(1, 2), form_ref=1.76, break_ref=1.76,
                r_inf=16.0)
    e = stepped("h3", [mass_au("H")] * 3, h3_collinear(), nbeads, 5, 0, thermostat="andersen")
    e.set_umbrella(centers=0.9, kforce=0.0, **mech)
    e.run(1)
    q, _, f, _, _ = e.get_state()
    _, want = egrad_h3(q.reshape(-1, 3, 3))
    rest = f - want.reshape(f.shape)            # the bias, one vector for all beads of a trajectory
    assert np.abs(rest - rest[:, :1]).max() <= 1e-15
    e.close()
    x, length = water_box(4, seed=3)
    w = WaterBox(4, box=[length] * 3, coul_cut=3.0)
    e = stepped(w, w.mass, x, nbeads, 2, 0)
    e.run(1)
    q, _, f, _, _ = e.get_state()
    _, want = w.egrad(q.reshape(-1, 12, 3))
    assert np.array_equal(f.reshape(want.shape), want)
    e.close()
