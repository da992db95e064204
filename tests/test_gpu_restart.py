"""GPU: a state that was saved and set again continues as the run it comes from.

Thermostats that draw leave momenta that differ between beads j and P - j; the step works
on their symmetric part alone, rounded as the state in between has it. So an engine that
receives another's state at the same step ends where that one does, bit for bit, and so
does a run that is read and set back after every step, for runs that end on a draw and
between draws, through cr_engine_run and through the host-buffer step."""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr, dt_fs_to_au
from caracal_gb300.workloads import ch4h_md_config, h3_config
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
CONFIG = {"h3": h3_config, "ch4h": ch4h_md_config}


def engine(pes, nbeads, ntraj, thermostat, precision="fp64", seed=4, sigma=0.02):
    wl = CONFIG[pes]()
    e = RPMDEngine(pes, wl.mass, nbeads, ntraj, wl.dt_au, beta=wl.beta, thermostat=thermostat, andersen_step=3,
                   pile_tau0_au=dt_fs_to_au(100.0), transrot=True, precision=precision, seed=seed)
    e.init_positions(wl.q0, float(angstrom_to_bohr(sigma)))
    e.init_momenta()
    e.compute_forces()
    return e


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("thermostat", ["andersen", "pile", "none"])
@pytest.mark.parametrize("pes,nbeads,ntraj,precision", [("h3", 3, 7, "fp64"), ("h3", 16, 5, "mixed"), ("h3", 16, 700, "fp64"),
                                                        ("ch4h", 7, 9, "fp64"), ("ch4h", 32, 20, "mixed")])
def test_state_moves_between_engines(require_gpu, pes, nbeads, ntraj, precision, thermostat):
    for n in (1, 3, 5):  # Andersen: between two draws, on one, past it
        a = engine(pes, nbeads, ntraj, thermostat, precision)
        b = engine(pes, nbeads, ntraj, thermostat, precision, sigma=0.03)  # another run, to the same step
        a.run(n)
        b.run(n)
        q, p, f, _, _ = a.get_state()
        b.set_state(q, p, f)
        a.run(5)
        b.run(5)
        assert same(a.get_state(), b.get_state()), n
        a.close()
        b.close()


@pytest.mark.parametrize("thermostat", ["andersen", "pile"])
@pytest.mark.parametrize("nbeads,ntraj", [(5, 3), (16, 200), (33, 4)])
def test_host_steps_are_the_run(require_gpu, nbeads, ntraj, thermostat):
    a, b = engine("h3", nbeads, ntraj, thermostat), engine("h3", nbeads, ntraj, thermostat)
    q, p, f, _, _ = b.get_state()
    a.run(8)
    for _ in range(8):
        b.step_host(q, p, f)
    want = a.get_state()
    assert same((q, p, f), want[:3])
    a.close()
    b.close()


@pytest.mark.parametrize("nbeads", [3, 4, 8, 16, 65])
def test_pile_momenta_of_every_bead(require_gpu, nbeads):
    """The antisymmetric part itself: p of all beads after one and after three PILE steps."""
    wl, tau = h3_config(), dt_fs_to_au(100.0)
    for n in (1, 3):
        e = engine("h3", nbeads, 6, "pile")
        cfg = orc.Config("h3", wl.mass, nbeads, wl.dt_au, wl.beta, thermostat="pile", andersen_step=3, pile_tau0=tau,
                         transrot=True, seed=4)
        q, p = orc.init_positions(cfg, 6, wl.q0, float(angstrom_to_bohr(0.02))), orc.init_momenta(cfg, 6)
        f, _ = orc.init_forces(cfg, q)
        e.run(n)
        q, p, f, _, _ = orc.run(cfg, q, p, f, n)
        assert rel_err(e.get_state()[1], p) <= (1e-12 if n == 1 else 1e-11)
        e.close()
