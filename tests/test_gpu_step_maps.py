"""GPU: the persistent step kernel's fixed-point linear maps and carried beads.

The free ring polymer and the PILE maps run in block fixed point on the
distinct beads of each ring polymer; folds, guard bits and table shapes change
with the bead count's parity and size, and thermostats that draw add an
antisymmetric part to the momenta at the end of a run.  Every such case
against the oracle at the repository's bars: 1e-12 after one step, 1e-9 after
twenty.  A run in pieces must be the run in one, bit for bit."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au, nose_q_to_au
from caracal_gb300.workloads import h3_collinear
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
KW = dict(andersen_step=4, transrot=True, seed=21)


def pair(nbeads, ntraj, thermostat, nm_mode=0):
    dt, beta, sig = dt_fs_to_au(0.1), beta_from_kelvin(300.0), float(angstrom_to_bohr(0.02))
    tau, nq = dt_fs_to_au(100.0), nose_q_to_au(100.0, 0.1)
    e = RPMDEngine("h3", [mass_au("H")] * 3, nbeads, ntraj, dt, beta=beta, thermostat=thermostat, pile_tau0_au=tau,
                   nose_q_au=nq, nm_mode=nm_mode, **KW)
    e.init_positions(h3_collinear(), sig)
    e.init_momenta()
    e.compute_forces()
    cfg = orc.Config("h3", [mass_au("H")] * 3, nbeads, dt, beta, thermostat=thermostat, pile_tau0=tau, nose_q=nq,
                     nm_mode=nm_mode, **KW)
    q = orc.init_positions(cfg, ntraj, h3_collinear(), sig)
    p = orc.init_momenta(cfg, ntraj)
    f, _ = orc.init_forces(cfg, q)
    return e, cfg, q, p, f


@pytest.mark.parametrize("thermostat", ["none", "andersen", "pile", "nhc"])
@pytest.mark.parametrize("nbeads", [1, 2, 3, 6, 7, 12, 33, 64, 127, 128])
def test_bead_counts_match_oracle(require_gpu, nbeads, thermostat):
    T = 3
    e, cfg, q, p, f = pair(nbeads, T, thermostat)
    vnh = np.zeros((T, 4))
    for n, bar in ((1, 1e-12), (19, 1e-9)):
        e.run(n)
        qg, pg, fg, eg, st = e.get_state()
        q, p, f, eo, so = orc.run(cfg, q, p, f, n, istep0=0 if n == 1 else 1, vnh=vnh)
        assert not st.any() and not so.any()
        errs = [rel_err(a, b) for a, b in ((qg, q), (pg, p), (fg, f), (eg, eo))]
        print(nbeads, thermostat, n, errs)
        assert max(errs) <= bar
    e.close()


@pytest.mark.parametrize("thermostat", ["andersen", "pile"])
@pytest.mark.parametrize("nbeads,nm_mode", [(5, 0), (16, 0), (6, 1)])
def test_a_run_in_pieces(require_gpu, nbeads, nm_mode, thermostat):
    a, b = pair(nbeads, 5, thermostat, nm_mode)[0], pair(nbeads, 5, thermostat, nm_mode)[0]
    a.run(12)
    for n in (1, 3, 4, 4):
        b.run(n)
    for x, y in zip(a.get_state(), b.get_state()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
