"""GPU: an H3 bead's energy and gradient do not depend on its batch.

Small batches take four lanes per bead, larger ones a thread each; the surface's source
decides every rounding, so both forms and both kernels give the same bits. Gradient calls
on either side of the line, and an ensemble stepped as a whole (more than the line's 4864
beads) and in parts with the trajectories' own noise keys."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine, egrad_h3
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au
from caracal_gb300.workloads import h3_collinear

pytestmark = pytest.mark.gpu


def beads(n):
    rng = np.random.default_rng(11)
    q = h3_collinear() + 0.3 * rng.standard_normal((n, 3, 3))
    q[::3, 1] = q[::3, 0] + 0.45 * rng.standard_normal((len(q[::3]), 3))  # compact ones among them
    return q


@pytest.mark.parametrize("n", [1, 9, 4864])
def test_gradient_calls(require_gpu, n):
    q = beads(9000)
    V, g = egrad_h3(q)
    v1, g1 = egrad_h3(q[:n])
    assert np.isfinite(V).all() and np.array_equal(v1, V[:n]) and np.array_equal(g1, g[:n])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("thermostat", ["none", "andersen", "pile"])
def test_ensemble_in_parts(require_gpu, precision, thermostat):
    T, P = 600, 16  # 5400 distinct beads
    def engine(traj0, ntraj):
        e = RPMDEngine("h3", [mass_au("H")] * 3, P, ntraj, dt_fs_to_au(0.1), beta=beta_from_kelvin(300.0),
                       thermostat=thermostat, andersen_step=3, pile_tau0_au=dt_fs_to_au(100.0), precision=precision,
                       seed=5, traj0=traj0)
        e.init_positions(h3_collinear(), float(angstrom_to_bohr(0.02)))
        e.init_momenta()
        e.compute_forces()
        e.run(10)
        out = e.get_state()
        e.close()
        return out
    whole = engine(0, T)
    for t0, n in ((0, 1), (1, 299), (300, 300)):
        for x, y in zip(engine(t0, n), whole):
            assert np.array_equal(x, y[t0:t0 + n])
