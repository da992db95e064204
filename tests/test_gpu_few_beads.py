"""GPU: ring polymers of one to four beads.

Up to two carried beads transrot is summed by a thread per trajectory about the
reference's centre; beyond, from moments. Every surface shape (one thread per bead, four
lanes) and more trajectories than a block holds, against the oracle at the one-step bar
(1e-12). With one bead that centre is the centre of mass, and a molecule 300 bohr away from
the origin is held to the same bar: about the centre it loses R/r = 150 roundings (3e-14),
about the origin (R/r)^2. (With more beads the reference's centre, 1/P of it, is off the
molecule itself, so that there is no such bar.)"""
import numpy as np
import pytest

from caracal_gb300 import RPMDEngine
from caracal_gb300.units import angstrom_to_bohr
from caracal_gb300.workloads import ch4h_md_config, ch4oh_md_config, oh3_config
from conftest import rel_err
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
CONFIG = {"oh3": oh3_config, "ch4h": ch4h_md_config, "ch4oh": ch4oh_md_config}


@pytest.mark.parametrize("pes,ntraj", [("oh3", 3), ("oh3", 300), ("ch4h", 130), ("ch4oh", 5)])
@pytest.mark.parametrize("nbeads,away", [(1, 0.0), (1, 300.0), (2, 0.0), (3, 0.0), (4, 0.0)])
def test_few_beads(require_gpu, pes, ntraj, nbeads, away):
    wl, sig = CONFIG[pes](), float(angstrom_to_bohr(0.02))
    q0 = np.asarray(wl.q0) + away * np.array([0.6, -0.48, 0.64])
    kw = dict(andersen_step=2, transrot=True, seed=3, thermostat="andersen")
    e = RPMDEngine(pes, wl.mass, nbeads, ntraj, wl.dt_au, beta=wl.beta, **kw)
    e.init_positions(q0, sig)
    e.init_momenta()
    e.compute_forces()
    cfg = orc.Config(pes, wl.mass, nbeads, wl.dt_au, wl.beta, **kw)
    q, p = orc.init_positions(cfg, ntraj, q0, sig), orc.init_momenta(cfg, ntraj)
    f, _ = orc.init_forces(cfg, q)
    for n in range(2):  # a step without and one with a draw
        e.run(1)
        qg, pg, fg, eg, st = e.get_state()
        q, p, f, eo, so = orc.run(cfg, q, p, f, 1, istep0=n)
        assert not st.any() and not so.any()
        errs = [rel_err(a, b) for a, b in ((qg, q), (pg, p), (fg, f), (eg, eo))]
        assert max(errs) <= 1e-12, errs
    e.close()


@pytest.mark.parametrize("pes,per_bead", [("oh3", (1, 2, 4)), ("ch4h", (1,))])
@pytest.mark.parametrize("nbeads", [1, 2, 3])
def test_shapes_agree(require_gpu, pes, per_bead, nbeads):
    """A trajectory by four lanes where the block has the threads, else by one: the same bits."""
    wl, T, group = CONFIG[pes](), 150, 1 << (nbeads - 1).bit_length()
    out = []
    for tpb in per_bead:
        for groups in (1, 7, 40, 64):
            block = groups * group * tpb
            if block > 256:
                continue
            e = RPMDEngine(pes, wl.mass, nbeads, T, wl.dt_au, beta=wl.beta, thermostat="andersen", andersen_step=3, seed=3)
            e.init_positions(wl.q0, float(angstrom_to_bohr(0.02)))
            e.init_momenta()
            e.compute_forces()
            e.set_launch(block, tpb)
            e.run(10)
            out.append(e.get_state())
            e.close()
    assert len(out) > 2 and all(np.array_equal(x, y) for o in out[1:] for x, y in zip(o, out[0]))
