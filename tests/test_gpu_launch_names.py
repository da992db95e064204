"""GPU: what the engine reports as its launch shape can be set.

The step kernel's blocks hold U = P/2 + 1 beads per trajectory where the API counts
next_pow2(P) threads, so more trajectories may fit a block than a nominal 256 threads
name.  For bead counts on either side of the powers of two: the built-in choice and the
autotuner's are set again as reported and give the same launch, and the reported grid and
block are those of the launch."""
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr
from caracal_gb300.workloads import ch4h_md_config, h3_config, oh3_config

pytestmark = pytest.mark.gpu
CONFIG = {"h3": h3_config, "ch4h": ch4h_md_config, "oh3": oh3_config}


def shape(e):
    info = e.launch_info()
    return e.launch(), info["grid"], info["block"], info["smem_bytes"]


def check(e, ntraj, nbeads):
    (block, blocks, tpb), grid, threads, _ = was = shape(e)
    assert 1 <= block <= 256 and block % ((1 << (nbeads - 1).bit_length()) * tpb) == 0
    assert blocks == grid and threads <= 128 and threads % 32 == 0
    distinct = nbeads // 2 + 1
    assert grid * (threads // distinct) >= ntraj  # every trajectory has its place
    e.set_launch(block, tpb)
    assert shape(e) == was


@pytest.mark.parametrize("pes,ntraj", [("h3", 9), ("h3", 3000), ("oh3", 1500), ("ch4h", 700)])
@pytest.mark.parametrize("nbeads", [1, 4, 5, 12, 17, 24, 33, 100])
def test_reported_shape_can_be_set(require_gpu, pes, ntraj, nbeads):
    wl = CONFIG[pes]()
    e = RPMDEngine(pes, wl.mass, nbeads, ntraj, wl.dt_au, beta=wl.beta, thermostat="andersen", precision="mixed", seed=1)
    e.init_positions(wl.q0, float(angstrom_to_bohr(0.01)))
    e.init_momenta()
    e.compute_forces()
    check(e, ntraj, nbeads)
    block, tpb, _ = e.autotune(1)
    assert e.launch()[::2] == (block, tpb)
    check(e, ntraj, nbeads)
    e.close()
