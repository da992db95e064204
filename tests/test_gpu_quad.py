"""GPU: four lanes per bead on the XH4 surfaces, and the free ring polymer by
fast transforms.

A quad's shuffles need whole warps, so a batch's last warp repeats a bead
without storing it: every bead of a ragged batch must be the bead alone, bit
for bit.  The fast transforms serve 32 and 64 beads; against the oracle at the
repository's bars (1e-12 after one step, 1e-9 after twenty)."""
import numpy as np
import pytest

import caracal_gb300 as cr
from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au
from caracal_gb300.workloads import h3_collinear
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def xh4(n_atoms, n, seed):
    q0 = np.array([[2.1, 0.0, 0.0], [0.0, 0.0, 0.0], [-0.7, 1.9, 0.1], [-0.7, -0.9, 1.7], [-0.6, -1.0, -1.7],
                   [4.4, 0.1, 0.0], [5.0, 1.6, 0.2]])[:n_atoms]
    return q0 + 0.1 * np.random.default_rng(seed).standard_normal((n, n_atoms, 3))


@pytest.mark.parametrize("pes,n_atoms", [("ch4h", 6), ("ch4oh", 7), ("geh4oh", 7)])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 33])
def test_ragged_batches(require_gpu, pes, n_atoms, n):
    f = getattr(cr, "egrad_" + pes)
    q = xh4(n_atoms, n, n)
    V, g = f(q)
    for i in range(n):
        v1, g1 = f(q[i])
        assert v1[0] == V[i] and np.array_equal(g1[0], g[i])


@pytest.mark.parametrize("nbeads", [32, 64])
def test_fast_ring_matches_oracle(require_gpu, nbeads):
    T, kw = 3, dict(andersen_step=4, transrot=True, seed=21, thermostat="andersen")
    dt, beta, sig = dt_fs_to_au(0.1), beta_from_kelvin(300.0), float(angstrom_to_bohr(0.02))
    e = RPMDEngine("h3", [mass_au("H")] * 3, nbeads, T, dt, beta=beta, **kw)
    e.init_positions(h3_collinear(), sig)
    e.init_momenta()
    e.compute_forces()
    cfg = orc.Config("h3", [mass_au("H")] * 3, nbeads, dt, beta, **kw)
    q, p = orc.init_positions(cfg, T, h3_collinear(), sig), orc.init_momenta(cfg, T)
    f, _ = orc.init_forces(cfg, q)
    for n, bar, at in ((1, 1e-12, 0), (19, 1e-9, 1)):
        e.run(n)
        got = e.get_state()[:4]
        q, p, f, eo, so = orc.run(cfg, q, p, f, n, istep0=at)
        errs = [rel_err(a, b) for a, b in zip(got, (q, p, f, eo))]
        print(nbeads, n, errs)
        assert not so.any() and max(errs) <= bar
    e.close()
