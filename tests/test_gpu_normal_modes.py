"""GPU: orthonormal normal modes (nm_mode 1) in the persistent step kernel.

All beads are carried and the maps are circulants, in fixed point: bead counts from one
to the most, odd and even, with and without a thermostat that draws, against the oracle
at the repository's bars (1e-12 after one step, 1e-9 after twenty)."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr, dt_fs_to_au, nose_q_to_au
from caracal_gb300.workloads import ch4h_md_config, h3_config
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
CONFIG = {"h3": h3_config, "ch4h": ch4h_md_config}


@pytest.mark.parametrize("thermostat", ["none", "andersen", "pile", "nhc"])
@pytest.mark.parametrize("pes,nbeads", [("h3", 1), ("h3", 2), ("h3", 5), ("h3", 16), ("h3", 33), ("h3", 100), ("h3", 127),
                                        ("h3", 128), ("ch4h", 7), ("ch4h", 32), ("ch4h", 128)])
def test_circulants_match_oracle(require_gpu, pes, nbeads, thermostat):
    wl, T, sig = CONFIG[pes](), 3, float(angstrom_to_bohr(0.02))
    tau, nq = dt_fs_to_au(100.0), nose_q_to_au(100.0, 0.1)
    kw = dict(andersen_step=4, transrot=True, seed=8, thermostat=thermostat, nm_mode=1)
    e = RPMDEngine(pes, wl.mass, nbeads, T, wl.dt_au, beta=wl.beta, pile_tau0_au=tau, nose_q_au=nq, **kw)
    e.init_positions(wl.q0, sig)
    e.init_momenta()
    e.compute_forces()
    cfg = orc.Config(pes, wl.mass, nbeads, wl.dt_au, wl.beta, pile_tau0=tau, nose_q=nq, **kw)
    q, p = orc.init_positions(cfg, T, wl.q0, sig), orc.init_momenta(cfg, T)
    f, _ = orc.init_forces(cfg, q)
    vnh = np.zeros((T, 4))
    for n, bar in ((1, 1e-12), (19, 1e-9)):
        e.run(n)
        qg, pg, fg, eg, st = e.get_state()
        q, p, f, eo, so = orc.run(cfg, q, p, f, n, istep0=0 if n == 1 else 1, vnh=vnh)
        assert not st.any() and not so.any()
        errs = [rel_err(a, b) for a, b in ((qg, q), (pg, p), (fg, f), (eg, eo))]
        assert max(errs) <= bar, errs
    e.close()
