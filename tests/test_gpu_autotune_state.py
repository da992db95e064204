"""GPU: the autotuner's trial runs leave no trace.

A run's last bits do not depend on the launch shape, and the trials restore all
that the next run reads (the momentum parts of a thermostat's last draw
included), so an engine that was tuned between two runs must end where one that
was not ends, bit for bit."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au, nose_q_to_au
from caracal_gb300.workloads import h3_collinear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thermostat", ["pile", "andersen", "nhc", "none"])
@pytest.mark.parametrize("nbeads", [5, 16])
def test_tuned_run_is_the_run(require_gpu, nbeads, thermostat):
    ends = []
    for tune in (False, True):
        e = RPMDEngine("h3", [mass_au("H")] * 3, nbeads, 7, dt_fs_to_au(0.1), beta=beta_from_kelvin(300.0),
                       thermostat=thermostat, andersen_step=3, pile_tau0_au=dt_fs_to_au(100.0),
                       nose_q_au=nose_q_to_au(100.0, 0.1), transrot=True, seed=4)
        e.init_positions(h3_collinear(), float(angstrom_to_bohr(0.02)))
        e.init_momenta()
        e.compute_forces()
        e.run(3)
        if tune:
            e.autotune(4)
        e.run(8)
        ends.append(e.get_state())
        e.close()
    assert all(np.array_equal(x, y) for x, y in zip(*ends))
