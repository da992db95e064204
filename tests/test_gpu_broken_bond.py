"""GPU: XH4 surfaces, mixed form, with a broken X-H bond in line with another.

The in-plane bend of two bonds divides by the sine of their angle. A hydrogen that the
attacking atom has taken passes through the line of another bond, where FP32 rounds
1 - cos^2 to 0 although the force is finite (its stiffness is about 0 there): GeH4 + OH
trajectories became non-finite that way. Angles from 1e-2 rad off the line to none, on both
sides, against the plain form: the unit vectors' rounding (6e-8) over the sine, times the
bend's force (at most the largest force: CH4 + H keeps half of the stiffness with its H-H
distance of 1.5 Angstrom), on top of the form's own bar; in line itself finite."""
import ctypes

import numpy as np
import pytest
import torch

from caracal_gb300 import lib
from caracal_gb300 import _lib as L
from caracal_gb300.units import angstrom_to_bohr
from caracal_gb300.workloads import ch4h_dividing_surface, ch4oh_geometry, geh4oh_geometry

pytestmark = pytest.mark.gpu
SURFACES = {"ch4h": (L.CR_PES_CH4H, ch4h_dividing_surface), "ch4oh": (L.CR_PES_CH4OH, ch4oh_geometry),
            "geh4oh": (L.CR_PES_GEH4OH, geh4oh_geometry)}


def egrad(pes, q, precision):
    x = torch.as_tensor(np.ascontiguousarray(q), device="cuda")
    V, g = torch.empty(len(q), dtype=torch.float64, device="cuda"), torch.empty_like(x)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    L.check(lib().cr_egrad_device(pes, p(x), len(q), p(V), p(g), precision, ctypes.c_void_p(0)), "egrad")
    torch.cuda.synchronize()
    return V.cpu().numpy(), g.cpu().numpy()


@pytest.mark.parametrize("surface", list(SURFACES))
@pytest.mark.parametrize("side", [1.0, -1.0])
def test_broken_bond_in_line(require_gpu, surface, side):
    pes, geometry = SURFACES[surface]
    rng = np.random.default_rng(5)
    off = np.array([0.0, 1e-8, 1e-6, 1e-5, 1e-4, 2e-4, 1e-3, 1e-2])
    q = []
    for delta in off:
        x = np.array(geometry(), dtype=np.float64) + rng.normal(0, 0.03, (len(geometry()), 3))
        u = (x[2] - x[1]) / np.linalg.norm(x[2] - x[1])      # the bond to atom 2
        w = np.cross(u, rng.normal(size=3))
        w /= np.linalg.norm(w)
        r = np.linalg.norm(x[0] - x[1]) + float(angstrom_to_bohr(1.9))
        shift = x[1] + r * (side * np.cos(delta) * u + np.sin(delta) * w) - x[0]
        x[0] += shift                                        # the broken bond's hydrogen
        x[5:] += shift                                       # and what has taken it
        q.append(x)
    Vm, gm = egrad(pes, q, L.CR_PREC_MIXED)
    assert np.isfinite(Vm).all() and np.isfinite(gm).all()
    V, g = egrad(pes, q, L.CR_PREC_FP64)
    for b, delta in enumerate(off):
        if delta < 1e-6:
            continue  # the plain form's own 1 - cos^2 has no digits left
        err = np.abs(gm[b] - g[b]).max() / np.abs(g[b]).max()
        assert err <= 2e-7 + 6e-8 / delta, (delta, err)
