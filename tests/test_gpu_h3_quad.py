"""GPU: the H3 surface by four lanes per bead and by one.

Batches of up to 4864 beads take four lanes per bead, larger ones a thread each.
Ragged small batches, with compact geometries among them (a distance below
1.15 bohr), against the same beads in a large batch (the same operations up to the
contraction of products and sums: 1e-13) and against the oracle at its bar
(1e-12)."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine, egrad_h3
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au
from caracal_gb300.workloads import h3_collinear
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def beads(n):
    q = h3_collinear() + 0.2 * np.random.default_rng(6).standard_normal((n, 3, 3))
    q[::3, 1] = q[::3, 0] + np.array([0.6, 0.5, 0.4])  # 0.88 bohr: compact
    return q


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 4864, 4865])
def test_lanes_match_threads_and_oracle(require_gpu, n):
    q = beads(6000)
    V, g = egrad_h3(q)
    v1, g1 = egrad_h3(q[:n])
    assert rel_err(v1, V[:n]) <= 1e-13 and rel_err(g1, g[:n]) <= 1e-13
    vo, go = orc.egrad("h3", q[:min(n, 64)])
    assert rel_err(v1[:64], vo) <= 1e-12 and rel_err(g1[:64], go) <= 1e-12


@pytest.mark.parametrize("ntraj,nbeads", [(3, 5), (540, 16), (541, 16)])
def test_step_on_either_side_of_the_line(require_gpu, ntraj, nbeads):
    dt, beta, sig = dt_fs_to_au(0.1), beta_from_kelvin(300.0), float(angstrom_to_bohr(0.02))
    kw = dict(andersen_step=4, transrot=True, seed=21, thermostat="andersen")
    e = RPMDEngine("h3", [mass_au("H")] * 3, nbeads, ntraj, dt, beta=beta, **kw)
    e.init_positions(h3_collinear(), sig)
    e.init_momenta()
    e.compute_forces()
    cfg = orc.Config("h3", [mass_au("H")] * 3, nbeads, dt, beta, **kw)
    q, p = orc.init_positions(cfg, ntraj, h3_collinear(), sig), orc.init_momenta(cfg, ntraj)
    f, _ = orc.init_forces(cfg, q)
    e.run(1)
    got = e.get_state()[:4]
    q, p, f, eo, so = orc.run(cfg, q, p, f, 1)
    e.close()
    assert not so.any() and max(rel_err(a, b) for a, b in zip(got, (q, p, f, eo))) <= 1e-12
