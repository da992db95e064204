"""GPU: engines of one surface with different block sizes share its step kernel.

The kernel's limit on dynamic shared memory is the process's, not the engine's: an engine
that is created or prepared last must not lower it for another.  CH4 + H with 32 beads at
seven trajectories per block (99 KB) and at one (17 KB), in one batch with the larger
block first, and one after another around an engine's creation; states bit for bit those
of separate runs."""
import numpy as np
import pytest

from caracal_gb300 import RPMDBatch, RPMDEngine
from caracal_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def engine(ntraj, precision, block=0):
    wl = W.ch4h_md_config(ntraj=ntraj, nbeads=32)
    e = RPMDEngine("ch4h", wl.mass, 32, ntraj, wl.dt_au, beta=wl.beta, thermostat="andersen", andersen_step=3,
                   precision=precision, seed=ntraj)
    e.init_positions(wl.q0, wl.sigma_bohr)
    e.init_momenta()
    e.compute_forces()
    if block:
        e.set_launch(block)
    return e


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_classes_of_one_surface(require_gpu, precision):
    a = [engine(14, precision, 224), engine(3, precision)]
    b = [engine(14, precision, 224), engine(3, precision)]
    assert a[0].launch_info()["smem_bytes"] > 90 * 1024 > 48 * 1024 > a[1].launch_info()["smem_bytes"]
    batch = RPMDBatch(a, chunk_steps=2)
    batch.run(5)
    b[1].run(5)
    small = engine(1, precision)      # its creation tries small blocks last
    b[0].run(5)
    for x, y in zip(a, b):
        for u, v in zip(x.get_state(), y.get_state()):
            assert np.array_equal(u, v)
    batch.close()
    for e in a + b + [small]:
        e.close()
