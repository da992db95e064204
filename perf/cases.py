"""Performance cases of the RPMD engine: what its users have it do, through the public entry points.

The kinds, with the sizes of the package's own workloads, tests and benchmark:

  egrad           one call of a surface on host arrays, as Caracal's `gradient` makes it
  md              an ensemble of ring polymers started and stepped on an analytic surface (`dynamic`)
  umbrella        a chunk of umbrella sampling over all windows of a rate calculation (`calc_rate`)
  recross         the recrossing children of one parent and their transmission coefficient (`calc_rate`)
  qmdff           NVT steps of a molecule on a QMDFF force field, resident on the device
  qmdff_npt       the same in a periodic box under the Berendsen barostat
  force_matching  loss and parameter gradient of a QMDFF over a set of geometries
  adjoint         a short trajectory and the gradient of a loss of its end, forward and backward

The plain form ("fp64") returns FP64 arrays.  The mixed form evaluates the surface in FP32, so its
frames are kept in FP32, which is all that a program that chose that form can use of them.

`exact` restates the surfaces it needs (BKMP2 H3, CH4 + H, QMDFF) and Caracal's step as plain torch
in 64 bits, gradients by autograd.
"""
import ctypes
import math

import numpy as np
import torch

import caracal_gb300 as cr
from caracal_gb300 import qmdff as Q
from caracal_gb300 import workloads as W
from caracal_gb300.fit import QMDFFParams, TrajectoryAdjoint, force_matching, trajectory_engine
from caracal_gb300.units import angstrom_to_bohr, beta_from_kelvin, dt_fs_to_au, mass_au, nose_q_to_au

EGRAD = {"h3": cr.egrad_h3, "oh3": cr.egrad_oh3, "ch4h": cr.egrad_ch4h, "ch4oh": cr.egrad_ch4oh,
         "geh4oh": cr.egrad_geh4oh}
CONFIG = {"h3": W.h3_config, "oh3": W.oh3_config, "ch4h": W.ch4h_md_config, "ch4oh": W.ch4oh_md_config,
          "geh4oh": W.geh4oh_md_config}
# additions, multiplications, divisions and function calls of one bead's energy and gradient
BEAD_FLOPS = {"h3": 1350.0, "oh3": 1700.0, "ch4h": 13000.0, "ch4oh": 15000.0, "geh4oh": 15000.0}
JITTER = float(angstrom_to_bohr(0.01))


def qmdff_flops(nc):
    n = 3 * nc + 2
    return 30.0 * n * (n - 1) + 2100.0 * n


def unique_beads(nbeads):
    # Caracal's free ring-polymer map gives beads j and P - j the same positions
    return nbeads // 2 + 1


def listed():
    return [
        # the per-bead call that an unchanged Caracal makes: one ring polymer's beads, host arrays
        {"name": "h3_egrad_call", "kind": "egrad", "pes": "h3", "nbeads": 16},
        # the small ensemble of `dynamic`: latency of the step is all that counts
        {"name": "h3_pile_mixed", "kind": "md", "pes": "h3", "ntraj": 64, "nbeads": 16, "thermostat": "pile",
         "precision": "mixed", "steps": 100},
        # umbrella sampling as in the H + H2 rate example: 110 windows x 10 ring polymers
        {"name": "h3_umbrella_fp64", "kind": "umbrella", "pes": "h3", "ntraj": 1100, "nbeads": 16, "steps": 40,
         "precision": "fp64"},
        # the benchmark's configuration: children of one dividing-surface parent, both forms
        {"name": "ch4h_recross_mixed", "kind": "recross", "ntraj": 4096, "nbeads": 32, "steps": 40,
         "precision": "mixed"},
        {"name": "ch4h_recross_fp64", "kind": "recross", "ntraj": 1000, "nbeads": 32, "steps": 20,
         "precision": "fp64"},
        # a larger reaction, more beads
        {"name": "ch4oh_md_mixed", "kind": "md", "pes": "ch4oh", "ntraj": 512, "nbeads": 64,
         "thermostat": "andersen", "precision": "mixed", "steps": 40},
        # a bead count that is no power of two, plain form, four atoms
        {"name": "oh3_md_fp64", "kind": "md", "pes": "oh3", "ntraj": 1000, "nbeads": 24, "thermostat": "andersen",
         "precision": "fp64", "steps": 40},
        # the molecular workload: C20H42, both forms; the plain one with ragged sizes
        {"name": "qmdff_nvt_mixed", "kind": "qmdff", "nc": 20, "ntraj": 1024, "nbeads": 64,
         "thermostat": "andersen", "precision": "mixed", "steps": 4},
        {"name": "qmdff_nvt_fp64", "kind": "qmdff", "nc": 13, "ntraj": 100, "nbeads": 48, "thermostat": "andersen",
         "precision": "fp64", "steps": 4},
        # the same molecule in a 40 Angstrom box at 1 atm
        {"name": "qmdff_npt_mixed", "kind": "qmdff_npt", "nc": 20, "ntraj": 256, "nbeads": 64,
         "precision": "mixed", "steps": 4},
        # derivatives: a force-matching evaluation, and a trajectory's adjoint
        {"name": "qmdff_force_matching", "kind": "force_matching", "nc": 20, "geometries": 2000},
        {"name": "qmdff_adjoint", "kind": "adjoint", "nc": 20, "ntraj": 16, "nbeads": 16, "steps": 20, "every": 5},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["egrad", "md", "md", "md", "umbrella", "recross", "recross", "qmdff", "qmdff", "qmdff_npt",
                       "force_matching", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "egrad":
        return {"kind": kind, "pes": rng.choice(sorted(EGRAD)), "nbeads": _log_int(rng, 1, 4096)}
    if kind in ("md", "umbrella", "recross"):
        pes = "ch4h" if kind == "recross" else rng.choice(["h3", "ch4h"] if kind == "umbrella" else sorted(CONFIG))
        nbeads = rng.choice([4, 6, 8, 12, 15, 16, 24, 32, 48, 64])
        # about the bead-steps that the largest listed case has time for
        small = pes in ("h3", "oh3")
        beads = (3e6 if small else 4e6) if precision == "mixed" else (1.5e6 if small else 8e5)
        steps = _log_int(rng, 5, 60)
        ntraj = _log_int(rng, 1, max(1, min(4096, int(beads / (nbeads * steps)))))
        case = {"kind": kind, "pes": pes, "ntraj": ntraj, "nbeads": nbeads, "precision": precision, "steps": steps}
        if kind == "recross":
            del case["pes"]
        if kind == "md":
            case["thermostat"] = rng.choice(["none", "andersen", "andersen", "pile", "nose-hoover"])
        return case
    nc = rng.randint(4, 20)
    if kind == "force_matching":
        return {"kind": kind, "nc": nc, "geometries": _log_int(rng, 50, 2000)}
    if kind == "adjoint":
        return {"kind": kind, "nc": nc, "ntraj": _log_int(rng, 1, 16), "nbeads": rng.choice([2, 4, 6, 8, 12, 16]),
                "steps": rng.randint(4, 20), "every": rng.randint(2, 8)}
    nbeads, steps = rng.choice([1, 4, 8, 12, 16, 24, 32, 48, 64, 96]), rng.randint(2, 6)
    most = (4e10 if precision == "mixed" else 3e9) / qmdff_flops(nc) / (nbeads * steps)
    case = {"kind": kind, "nc": nc, "ntraj": _log_int(rng, 1, max(1, min(1024, int(most)))), "nbeads": nbeads,
            "precision": precision, "steps": steps}
    if kind == "qmdff":
        case["thermostat"] = rng.choice(["none", "andersen", "andersen", "pile"])
    return case


# ---- what a program holds before the call ------------------------------------------------------

class DeviceArray:
    """An engine's state array on the device (cr_engine_device_state) as torch sees it.  torch keeps this
    object as long as the tensor, and this object keeps the engine that owns the memory."""

    def __init__(self, owner, ptr):
        self.owner = owner
        shape = owner.shape
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": "<f8",
                                         "version": 2}


def device_state(eng):
    ptrs = [ctypes.c_void_p() for _ in range(3)]
    rc = cr.lib().cr_engine_device_state(eng._h, *[ctypes.byref(p) for p in ptrs])
    if rc:
        raise RuntimeError("cr_engine_device_state: status %d" % rc)
    return [torch.as_tensor(DeviceArray(eng, p.value), device="cuda") for p in ptrs]


def h3_window_geometry(xi):
    """Collinear H-H...H with the reaction coordinate about xi: from 0.74 / 4 Angstrom to the saddle."""
    s = min(max(xi, 0.0), 1.0)
    return W.h3_collinear(0.74 + 0.19 * s, 4.0 - 3.07 * s)


def start_geometry(case, seed):
    """The case's structure (natoms, 3) in bohr, slightly displaced: every seed has its own."""
    rng = np.random.default_rng(seed)
    pes = case.get("pes", "ch4h")
    q0 = W.ch4h_dividing_surface() if case["kind"] == "recross" else CONFIG[pes]().q0
    return q0 + rng.normal(0.0, 0.02, q0.shape)


def umbrella_input(case, seed):
    rng = np.random.default_rng(seed)
    T, P = case["ntraj"], case["nbeads"]
    if case["pes"] == "h3":
        ts = W.h3_collinear(0.93, 0.93)
        mech = dict(reac1=[1, 2], reac2=[3], bond_form=(2, 3), bond_break=(1, 2), r_inf=16.0, xi_ideal=1.0,
                    form_ref=float(np.linalg.norm(ts[1] - ts[2])), break_ref=float(np.linalg.norm(ts[0] - ts[1])))
        centers = np.linspace(0.4, 1.05, T) if T > 1 else np.array([1.0])
        q0 = np.stack([h3_window_geometry(c) for c in centers])
    else:
        mech = W.ch4h_recross_definition(W.ch4h_dividing_surface())
        centers = np.linspace(0.95, 1.05, T) if T > 1 else np.array([1.0])
        q0 = np.repeat(W.ch4h_dividing_surface()[None], T, axis=0)
    wl = CONFIG[case["pes"]]()
    q = q0[:, None] + rng.normal(0.0, 0.03, (T, P) + q0.shape[1:])
    beta = beta_from_kelvin(300.0)
    p = rng.normal(0.0, 1.0, q.shape) * np.sqrt(wl.mass[:, None] * P / beta)
    return dict(mass=wl.mass, beta=beta, dt=dt_fs_to_au(0.1), mech=mech, centers=centers, kforce=0.2, q=q, p=p)


def qmdff_input(case, seed):
    ff = Q.alkane(nc=case["nc"])
    mass = np.array([mass_au("C" if z == 6 else "H") for z in ff.at])
    T, P = case["ntraj"], case["nbeads"]
    beta = beta_from_kelvin(300.0)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    shape = (T, P, ff.n, 3)
    normal = lambda: torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64)  # noqa: E731
    q = _t(ff.xyz) + 0.03 * normal()
    p = normal() * _t(np.sqrt(mass * P / beta))[:, None]
    return dict(ff=ff, mass=mass, beta=beta, dt=dt_fs_to_au(0.5), q=q, p=p)


def matching_input(case, seed):
    rng = np.random.default_rng(seed)
    ff = Q.alkane(nc=case["nc"])
    params = QMDFFParams(ff)
    theta = params.theta() * rng.uniform(0.9, 1.1, params.size)
    xyz = ff.xyz + rng.normal(0.0, 0.05, (case["geometries"], ff.n, 3))
    f_ref = rng.normal(0.0, 0.02, xyz.shape)
    return ff, params, theta, xyz, f_ref


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "egrad":
        rng = np.random.default_rng(seed)
        q0 = CONFIG[case["pes"]]().q0
        s["q"] = q0 + rng.normal(0.0, 0.05, (case["nbeads"],) + q0.shape)
    elif kind == "md":
        wl = CONFIG[case["pes"]](ntraj=case["ntraj"], nbeads=case["nbeads"])
        s["q0"] = start_geometry(case, seed)
        s["eng"] = cr.RPMDEngine(case["pes"], wl.mass, wl.nbeads, wl.ntraj, wl.dt_au, beta=wl.beta,
                                 thermostat=case["thermostat"], andersen_step=wl.andersen_step,
                                 pile_tau0_au=wl.pile_tau0_au, nose_q_au=nose_q_to_au(100.0, wl.dt_fs),
                                 precision=case["precision"], seed=seed & 0xFFFFFFFF)
    elif kind == "umbrella":
        u = umbrella_input(case, seed)
        eng = cr.RPMDEngine(case["pes"], u["mass"], case["nbeads"], case["ntraj"], u["dt"], beta=u["beta"],
                            thermostat="andersen", andersen_step=70, precision=case["precision"],
                            seed=seed & 0xFFFFFFFF)
        eng.set_umbrella(centers=u["centers"], kforce=u["kforce"], nbins=60, lo=-0.1, hi=1.2, **u["mech"])
        eng.set_state(u["q"], u["p"])
        eng.umbrella_sampling(True)
        s["eng"] = eng
    elif kind == "recross":
        wl = W.ch4h_config(ntraj=case["ntraj"], nbeads=case["nbeads"])
        q0 = start_geometry(case, seed)
        s["parent"] = np.repeat(q0[None], wl.nbeads, axis=0)
        s["parent"] = s["parent"] + np.random.default_rng(seed + 1).normal(0.0, JITTER, s["parent"].shape)
        s["eng"] = cr.RPMDEngine("ch4h", wl.mass, wl.nbeads, wl.ntraj, wl.dt_au, beta=wl.beta, transrot=False,
                                 precision=case["precision"], seed=seed & 0xFFFFFFFF)
        s["eng"].set_recross(max_steps=case["steps"], **W.ch4h_recross_definition(W.ch4h_dividing_surface()))
    elif kind in ("qmdff", "qmdff_npt"):
        u = qmdff_input(case, seed)
        s["ff"] = cr.QMDFFForceField(u["ff"])
        if kind == "qmdff_npt":
            s["ff"].set_periodic([40.0] * 3, 50.0, 10.0)
        s["eng"] = cr.RPMDEngine(s["ff"], u["mass"], case["nbeads"], case["ntraj"], u["dt"], beta=u["beta"],
                                 thermostat=case.get("thermostat", "andersen"), andersen_step=70,
                                 pile_tau0_au=dt_fs_to_au(100.0), precision=case["precision"],
                                 seed=seed & 0xFFFFFFFF)
        if kind == "qmdff_npt":
            s["eng"].set_npt(1.0)
        s["eng"].set_state(u["q"].cpu().numpy(), u["p"].cpu().numpy())
    elif kind == "force_matching":
        _, s["params"], s["theta"], s["xyz"], s["f_ref"] = matching_input(case, seed)
    else:
        u = qmdff_input(case, seed)
        s["params"] = QMDFFParams(u["ff"])
        s["q0"], s["p0"] = u["q"].cpu().numpy(), u["p"].cpu().numpy()
        s["eng"], s["ff"] = trajectory_engine(s["params"], s["params"].theta(), u["mass"], case["nbeads"],
                                              case["ntraj"], u["dt"], u["beta"], s["q0"], s["p0"])
        s["adj"] = TrajectoryAdjoint(s["eng"], case["steps"], case["every"])
    if "eng" in s and kind != "adjoint":
        s["dev"] = device_state(s["eng"])
    return s


def frames(s):
    """q, p and dV/dq on the device, in the precision that the case's form has."""
    if s["case"]["precision"] == "mixed":
        return [x.float() for x in s["dev"]]
    return list(s["dev"])


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "egrad":
        return list(EGRAD[case["pes"]](s["q"]))
    if kind == "force_matching":
        loss, grad = force_matching(s["params"], s["theta"], s["xyz"], s["f_ref"])
        return [float(loss), grad]
    eng = s["eng"]
    if kind == "adjoint":
        eng.set_state(s["q0"], s["p0"])
        s["adj"].forward()
        q, p = eng.get_state()[:2]
        grad, dq0, dp0 = s["adj"].backward(q - s["q0"], p * 1e-3)
        return [q, p, grad, dq0, dp0]
    if kind == "md":
        eng.init_positions(s["q0"], JITTER)
        eng.init_momenta()
        eng.compute_forces()
        eng.run(case["steps"])
        return frames(s)
    if kind == "umbrella":
        eng.run(case["steps"])
        xs, x2, hist = eng.umbrella_stats(reset=True)
        return frames(s) + ([xs, x2, hist] if case["precision"] == "fp64" else [])
    if kind == "recross":
        eng.init_children(s["parent"])
        eng.run(case["steps"])
        num, den, weights = eng.kappa(case["steps"])
        return frames(s) + [num, den, weights]
    eng.run(case["steps"])
    if kind == "qmdff_npt":
        box, pressure, _ = eng.npt_state()
        return frames(s) + [box.astype(np.float32), pressure.astype(np.float32)] if case["precision"] == "mixed" \
            else frames(s) + [box, pressure]
    return frames(s)


def work(case):
    kind = case["kind"]
    if kind == "egrad":
        n = CONFIG[case["pes"]]().q0.size
        return {"bytes": 8.0 * case["nbeads"] * (2 * n + 1), "flops": case["nbeads"] * BEAD_FLOPS[case["pes"]]}
    if kind == "force_matching":
        n, G = 3 * case["nc"] + 2, case["geometries"]
        # a gradient of every geometry, and its product with every parameter's derivative
        return {"bytes": 8.0 * G * 6 * n, "flops": 2.0 * G * qmdff_flops(case["nc"])}
    P, T, steps = case["nbeads"], case["ntraj"], case["steps"]
    if kind in ("md", "umbrella", "recross"):
        pes = case.get("pes", "ch4h")
        n3, flops = CONFIG[pes]().q0.size, BEAD_FLOPS[pes]
    else:
        n3, flops = 3 * (3 * case["nc"] + 2), qmdff_flops(case["nc"])
    # q, p and the gradient in and out once; per step the surface on the beads that differ, the
    # free ring polymer by fast transforms and the kicks, thermostat and centre-of-mass sums
    step = unique_beads(P) * (flops + n3 * (10.0 * math.log2(P + 1) + 20.0))
    if kind == "adjoint":  # forward, its repetition from the checkpoints, Hessian-vector and parameter products
        step *= 5.0
    return {"bytes": 8.0 * 6 * T * P * n3, "flops": T * steps * step}


# ---- 64-bit values ------------------------------------------------------------------------------

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(x, dtype=torch.float64, device=DEV)


def _r4(x):
    return float(np.float32(x))  # a REAL(4) literal of the published code, widened


def _h2_curves(R):
    """Singlet and triplet H2 curves of BKMP2."""
    a = [_r4(x) for x in (0.03537359271649620, 2.013977588700072, -2.827452449964767, 2.713257715593500,
                          -2.792039234205731, 2.166542078766724, -1.272679684173909, 0.5630423099212294,
                          -0.1879397372273814, 0.04719891893374140, -0.008851622656489644, 0.001224998776243630)]
    a += [-1.227820520228028e-04, 8.638783190083473e-06, -4.036967926499151e-07, 1.123286608335365e-08,
          -1.406619156782167e-10]
    alpha = a[0] / R + sum(a[k] * R ** (k - 1) for k in range(1, 17))
    D, R0 = 0.160979391, 3.5284882
    e1 = (D * (torch.exp(alpha) - 1.0) ** 2 - D - 6.499027 / (R ** 6 + R0 ** 6)
          - 124.3991 / (R ** 4 + R0 ** 4) ** 2 - 3285.828 / (R ** 2 + R0 ** 2) ** 5)
    b1, b2, b3, b4, b5, b6 = (_r4(x) for x in (-0.0298546962, -23.9604445036, -42.5185569474, 2.0382390988,
                                               -11.5214861455, 1.5309487826))
    c1, c2, c3 = (_r4(x) for x in (-0.4106358351531854, -0.0770355790707090, 0.4303193846943223))
    far = b1 * (b2 + R + b3 * R * R + b5 * R ** (-b6)) * torch.exp(-b4 * R)
    d = R - 0.95
    near = e1 + c2 * d + c3 + torch.where(R > 0.95, c1 * d ** 3, torch.zeros_like(d))
    return e1, torch.where(R >= 1.15, far, near)


_VB = {  # VBNDA, VBNDB
    "a": [-.1838073394E+03, 0.1334593242E+02, -.2358129537E+00, -.4668193478E+01, 0.7197506670E+01,
          0.2162004275E+02, 0.2106294028E+02, 0.4242962586E+01, 0.4453505045E+01, -.1456918088E+00,
          -.1692657366E-01, 0.1279520698E+01, -.4898940075E+00, 0.1742295219E+03, 0.3142175348E+02,
          0.5152903406E+01],
    "b": [-.4765732725E+02, 0.3648933563E+01, -.7141145244E-01, 0.1002349176E-01, 0.9989856329E-02,
          -.4161953634E-02, 0.9075807910E-03, -.2693628729E+00, -.1399065763E-01, -.1417634346E-01,
          -.4870024792E-03, 0.1312231847E+00, -.4409850519E-01, 0.5382970863E+02, 0.4587102824E+01,
          0.1768550515E+01]}


def h3_energy(q):
    """BKMP2 H3 (Boothroyd et al. 1991, 1996) at q (..., 3, 3) where no distance is below 1.15 bohr (the
    compact corrections are left out; None is returned where one is)."""
    r = torch.stack([(q[..., 1, :] - q[..., 0, :]).norm(dim=-1), (q[..., 0, :] - q[..., 2, :]).norm(dim=-1),
                     (q[..., 2, :] - q[..., 1, :]).norm(dim=-1)], dim=-1)
    if bool((r < 1.15).any()):
        return None
    e1, e3 = _h2_curves(r)
    J = 0.5 * (e1 - e3)
    d = J - J.roll(1, dims=-1)
    V = 0.5 * (e1 + e3).sum(-1) - torch.sqrt(0.5 * (d * d).sum(-1) + 1.0e-12)
    r1, r2, r3 = r.unbind(-1)
    A = ((r1 - r2) * (r2 - r3) * (r3 - r1)).abs()
    s = r.sum(-1)
    k = [_r4(x) for x in (0.3788951192E-02, 0.1478100901E-02, -.1848513849E-03, 0.9230803609E-05,
                          -.1293180255E-06, 0.5237179303E+00, -.1112326215E-02)]
    V = V + A ** 2 * (k[1] + A * (k[2] + A * (k[3] + A * k[4]))) * torch.exp(-k[0] * s ** 3) \
        + k[6] * A ** 2 * torch.exp(-k[5] * s) / s
    c1 = (r1 ** 2 - r2 ** 2 - r3 ** 2) / (-2.0 * r2 * r3)
    c2 = (r2 ** 2 - r3 ** 2 - r1 ** 2) / (-2.0 * r3 * r1)
    c3 = (r3 ** 2 - r1 ** 2 - r2 ** 2) / (-2.0 * r1 * r2)
    csum = c1 + c2 + c3
    cos3 = sum((4.0 * c * c - 3.0) * c for c in (c1, c2, c3))
    b2 = 1.0 / r1 + 1.0 / r2 + 1.0 / r3
    b3 = (r2 - r1) ** 2 + (r3 - r2) ** 2 + (r1 - r3) ** 2
    x1, x2, x7 = torch.exp(-0.52 * s), torch.exp(-0.052 * s * s), torch.exp(-0.79 * s)
    for name, B in (("a", 1.0 - csum), ("b", 1.0 - (0.625 * cos3 + 0.375 * csum))):
        c = [_r4(x) for x in _VB[name]]
        V = V + B * (c[0] + c[1] * s + c[2] * s * s) * x1
        V = V + (c[3] * B ** 2 + c[4] * B ** 3 + c[5] * B ** 4 + c[6] * B ** 5) * x2
        V = V + b2 * (c[7] * B * x1 + c[8] * B ** 2 * x2)
        V = V + B * (b3 * (c[9] * x1 + c[10] * x2) + torch.sqrt(b3 + 1.0e-12) * (c[11] * x1 + c[12] * x2))
        V = V + B * (c[13] + c[14] * s + c[15] * s * s) * x7
    return V


def ch4h_energy(q):
    """CH4 + H (Corchado, Bravo, Espinosa-Garcia 2009), 10^5 J/mol, at q (..., 6, 3) in bohr."""
    x = q * 0.52918
    h = x[..., [2, 3, 4, 0], :]
    c, b = x[..., 1, :], x[..., 5, :]
    t = c[..., None, :] - h
    rch, rbh, rcb = t.norm(dim=-1), (b[..., None, :] - h).norm(dim=-1), (c - b).norm(dim=-1)
    u = t / rch[..., None]
    dx = rch - 1.08898
    sw = lambda a: 1.0 - torch.tanh(a)  # noqa: E731
    s1 = sw(1.5132681e-7 * dx * (rch + 4.3792246) ** 8)
    s2 = sw(1.9202402e-7 * dx * (rch + 12.323018) ** 6)
    s3 = sw(0.1475300 * dx * (rch + 2.9926300) ** 2)
    zero = torch.zeros_like(rch)
    sphi = torch.where(rch < 3.8, sw(0.5307000 * dx * torch.exp(0.4012200 * (rch - 1.9235100) ** 3)), zero)
    sth = torch.where(rch < 3.8, sw(0.9119800 * dx * torch.exp(0.3537500 * (rch - 1.8970500) ** 3)), zero)
    tau = math.acos(-1.0 / 3.0)

    def others(*idx):
        return [k for k in range(4) if k not in idx]

    def theta0(i, j):
        m, n = others(i, j)
        return tau + (tau - 0.5 * math.pi) * (sphi[..., i] * sphi[..., j] - 1.0) \
            + (tau - 2.0 * math.pi / 3.0) * (sth[..., m] * sth[..., n] - 1.0)

    # stretches: LEPS forms of C-H_i, C-H_b, H_b-H_i
    morse = lambda r, r0, a, d1, d3: (lambda e: (0.5 * (d1 * (e * e - 2 * e) + d3 * (e * e + 2 * e)),  # noqa: E731
                                                 0.5 * (d1 * (e * e - 2 * e) - d3 * (e * e + 2 * e))))(
        torch.exp(-a * (r - r0)))
    f = 0.041840
    ach = 1.78374 + 0.14201 * 0.5 * (torch.tanh(2.21773 * (rch.mean(-1) - 1.08898)) + 1.0)
    qcb, jcb = morse(rcb, 1.08898, 1.41732, 56.505 * f, 19.612 * f)
    V = torch.zeros_like(rcb)
    for i in range(4):
        qch, jch = morse(rch[..., i], 1.08898, ach, 111.266 * f, 48.96226 * f)
        qbh, jbh = morse(rbh[..., i], 0.74239, 1.9589, 108.382 * f, 38.42657 * f)
        V = V + qch + qcb + qbh - torch.sqrt(0.5 * ((jch - jcb) ** 2 + (jcb - jbh) ** 2 + (jbh - jch) ** 2))
    # out-of-plane bends: angle of each other bond to the plane normal of the three hydrogens
    fch3, hch3 = 0.0693700 * 6.022045, 0.1387400 * 6.022045
    for i in range(4):
        trio = [(i + 1) & 3, (i + 2) & 3, (i + 3) & 3]
        j, k, l = trio
        n = torch.linalg.cross(h[..., k, :] - h[..., j, :], h[..., l, :] - h[..., j, :])
        n = n / n.norm(dim=-1, keepdim=True)
        cosn = [-(n * u[..., m, :]).sum(-1) for m in trio]
        flips = sum((v.detach() > 0).to(torch.int64) for v in cosn)
        sgn = (1 - 2 * (flips % 2)).to(torch.float64)
        dl = [torch.acos(sgn * v) - theta0(i, m) for v, m in zip(cosn, trio)]
        swi = (1.0 - s3[..., i]) * s3[..., j] * s3[..., k] * s3[..., l]
        V = V + swi * (fch3 * sum(d ** 2 for d in dl) + hch3 * sum(d ** 4 for d in dl))
    # in-plane bends
    fk, ak = 0.4291400 * 6.022045, 0.1353000 * 6.022045
    a1 = 1.0 - torch.exp(-1.265960 * rbh ** 2)
    a2 = 0.000710 + 0.985920 * torch.exp(-2.785060 * (rbh - 0.74239) ** 2)
    f1 = a1 * torch.exp(-a2 * dx ** 2)
    for i in range(3):
        for j in range(i + 1, 4):
            m, n = others(i, j)
            k0 = (fk + ak) * s1[..., i] * s1[..., j] + ak * (s2[..., m] * s2[..., n] - 1.0)
            d = torch.acos((u[..., i, :] * u[..., j, :]).sum(-1)) - theta0(i, j)
            V = V + 0.5 * k0 * f1[..., i] * f1[..., j] * d * d
    return V


def grad_of(energy, q, scale=1.0):
    """Energies and gradients (times scale) of q (..., natoms, 3), by autograd in pieces."""
    flat = q.reshape(-1, *q.shape[-2:])
    E, G = [], []
    for x in flat.split(8192):
        x = x.detach().requires_grad_(True)
        e = energy(x)
        if e is None:
            return None
        G.append(torch.autograd.grad(e.sum(), x)[0] * scale)
        E.append(e.detach())
    return torch.cat(E).reshape(q.shape[:-2]), torch.cat(G).reshape(q.shape)


def surface(pes):
    # the published CH4 + H code has two unit factors: of its energy and of its gradient
    if pes == "h3":
        return lambda q: grad_of(h3_energy, q)
    return lambda q: (lambda r: (r[0] * 0.03812, r[1]))(grad_of(ch4h_energy, q, 0.0201723 / 0.52918))


class QMDFFEnergy:
    """The synthetic QMDFF's energy: stretches, damped bends and torsions, NCI pairs."""

    def __init__(self, ff, theta=None):
        ix = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int64) - 1, device=DEV)  # noqa: E731
        params = QMDFFParams(ff)
        self.theta = _t(params.theta() if theta is None else theta)
        nb, na, nt = params.nbond, params.nangl, params.ntors
        self.cut = (nb, nb + na, nb + na + nt)
        self.bond, self.angl, self.tors, self.nci = ix(ff.bond), ix(ff.angl), ix(ff.tors[:, :4]), ix(ff.nci[:, :2])
        self.vb, self.va, self.vt = _t(ff.vbond), _t(ff.vangl), _t(ff.vtors)
        self.rad = _t(Q.element_radii())[torch.as_tensor(np.asarray(ff.at), device=DEV) - 1]
        self.r0, self.c6, self.s42, self.zab, self.alp = (_t(v) for v in
                                                          Q.pair_parameters(ff, Q.ElementTables.caracal()))
        e1, e2 = Q.eps_factors()
        self.e1, self.e2 = _t(e1[ff.nci[:, 2]]), _t(e2[ff.nci[:, 2]])
        self.pairs = None  # set to a vector: the pairs' charge products as parameters

    def damp(self, i, j, v):
        rcut = _r4(_r4(3.0) * _r4(3.5710642)) * (self.rad[i] + self.rad[j]) ** 2
        return 1.0 / (1.0 + ((v * v).sum(-1) / rcut) ** 2)

    def __call__(self, x, theta=None):
        th = self.theta if theta is None else theta
        kb, ka, kt, qa = th[:self.cut[0]], th[self.cut[0]:self.cut[1]], th[self.cut[1]:self.cut[2]], th[self.cut[2]:]
        i, j = self.bond.T
        r = (x[:, i] - x[:, j]).norm(dim=-1)
        y = (self.vb[:, 0] / r) ** (self.vb[:, 2] / 2)
        E = (kb * (1.0 + y * y - 2.0 * y)).sum(-1)
        j, i, k = self.angl.T
        a, b = x[:, i] - x[:, j], x[:, k] - x[:, j]
        cosa = (a * b).sum(-1) / (a.norm(dim=-1) * b.norm(dim=-1))
        E = E + (ka * (cosa - torch.cos(self.va[:, 0])) ** 2 * self.damp(i, j, a) * self.damp(k, j, b)).sum(-1)
        i, j, k, l = self.tors.T
        a, b, c = x[:, j] - x[:, i], x[:, k] - x[:, j], x[:, l] - x[:, k]
        n1, n2 = torch.linalg.cross(a, b), torch.linalg.cross(b, c)
        phi = torch.atan2(b.norm(dim=-1) * ((a * n2).sum(-1)).abs(), (n1 * n2).sum(-1))
        p0, rn, ph, vn = self.vt[:, 0], self.vt[:, 2], self.vt[:, 3], self.vt[:, 4]
        ef = torch.erf(phi - math.pi)
        et = 0.5 * (1.0 - ef) * vn * (1.0 + torch.cos(rn * (phi - p0) + ph)) \
            + 0.5 * (1.0 + ef) * vn * (1.0 + torch.cos(rn * (phi + p0 - 2.0 * math.pi) + ph))
        E = E + (kt * et * self.damp(i, j, a) * self.damp(k, j, b) * self.damp(k, l, c)).sum(-1)
        i, j = self.nci.T
        r = (x[:, i] - x[:, j]).norm(dim=-1)
        disp = -self.c6 / (r ** 6 + self.r0 ** 6) - self.s42 * self.c6 / (r ** 8 + self.r0 ** 8)
        rep = torch.where(r < 25.0, self.zab * torch.exp(-self.alp * r) / r, torch.zeros_like(r))
        coul = torch.where(r <= 50.0, self.e1 * qa[i] * qa[j] / r, torch.zeros_like(r))
        return E + (self.e2 * (disp + rep) + coul).sum(-1)


def normals(seed, traj, bead, step, tag, n):
    """The engine's documented noise: Philox4x32-10 words (key seed, trajectory; counter quad, bead, step, tag),
    24-bit uniforms, Box-Muller.  traj and bead: integer arrays of one shape; returns (..., n)."""
    m32 = np.uint64(0xFFFFFFFF)
    out = np.zeros(traj.shape + (n + (-n) % 4,))
    for quad in range((n + 3) // 4):
        c = [np.full(traj.shape, quad, np.uint64), bead.astype(np.uint64), np.full(traj.shape, step, np.uint64),
             np.full(traj.shape, tag, np.uint64)]
        k0, k1 = np.full(traj.shape, seed, np.uint64), traj.astype(np.uint64)
        for _ in range(10):
            a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
            c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & m32, (a >> np.uint64(32)) ^ c[3] ^ k1, a & m32]
            k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m32, (k1 + np.uint64(0xBB67AE85)) & m32
        for half in range(2):
            u = ((c[2 * half] >> np.uint64(8)) + np.uint64(1)).astype(float) * 2.0 ** -24
            v = (c[2 * half + 1] >> np.uint64(8)).astype(float) * 2.0 ** -24
            rad = np.sqrt(-2.0 * np.log(u))
            out[..., 4 * quad + 2 * half] = rad * np.cos(2.0 * np.pi * v)
            out[..., 4 * quad + 2 * half + 1] = rad * np.sin(2.0 * np.pi * v)
    return out[..., :n]


def ring_map(P, beta, dt):
    """Caracal's free ring polymer at unit mass: q' = K1 q + K3 p / m, p' = K1 p + m K2 q."""
    j = np.arange(P)
    C = np.sqrt(1.0 / P) * np.cos(2.0 * np.pi * np.outer(j, j) / P)
    w = 2.0 * P / beta * np.sin(np.minimum(j, P - j) * np.pi / P)
    s = np.where(w > 0, np.sin(w * dt) / np.where(w > 0, w, 1.0), dt)
    return [_t(C @ np.diag(d) @ C) for d in (np.cos(w * dt), -w * np.sin(w * dt), s)]


def remove_motion(q, p, m, P):
    """Caracal's transrot with its total mass P^2 sum m."""
    tm = P * P * m.sum()
    v, mm = p / m[:, None], m[:, None]
    vt, xt = (v * mm).sum((1, 2)) / tm, (q * mm).sum((1, 2)) / tm
    L = (torch.linalg.cross(q, v) * mm).sum((1, 2)) - torch.linalg.cross(xt, vt) * tm
    d = q - xt[:, None, None]
    S = torch.einsum("tbai,tbaj,a->tij", d, d, m)
    inertia = torch.eye(3, dtype=S.dtype, device=S.device) * S.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None] - S
    w = torch.linalg.solve(inertia, L)
    v = v - vt[:, None, None] - torch.linalg.cross(w[:, None, None].expand_as(d), d)
    return v * mm


def step(q, p, f, m, K, dt, force, transrot):
    mm = m[:, None]
    p = p - 0.5 * dt * f
    mul = lambda A, x: torch.einsum("jl,tl...->tj...", A, x)  # noqa: E731
    q, p = mul(K[0], q) + mul(K[2], p) / mm, mul(K[0], p) + mm * mul(K[1], q)
    f = force(q)
    if f is None:
        return None
    p = p - 0.5 * dt * f
    if transrot:
        p = remove_motion(q, p, m, q.shape[1])
    return q, p, f


def exact(case, seed):
    kind = case["kind"]
    if kind == "egrad":
        if case["pes"] not in ("h3", "ch4h"):
            return None  # surfaces that fill a file of their own
        r = surface(case["pes"])(_t(prepare(case, seed)["q"]))
        return None if r is None else list(r)
    if kind == "force_matching":
        ff, params, theta, xyz, f_ref = matching_input(case, seed)
        th = _t(theta).requires_grad_(True)
        E = QMDFFEnergy(ff)
        loss, grad = 0.0, torch.zeros_like(th)
        for x, fr in zip(_t(xyz).split(500), _t(f_ref).split(500)):
            x = x.requires_grad_(True)
            g = torch.autograd.grad(E(x, th).sum(), x, create_graph=True)[0]
            part = ((g + fr) ** 2).sum() / len(xyz)
            grad = grad + torch.autograd.grad(part, th)[0]
            loss += float(part.detach())
        return [loss, grad]
    if kind == "adjoint":
        # the device's parameters are the force constants and each pair's charge product
        return None if case["ntraj"] * case["nbeads"] * case["steps"] > 6000 else _exact_adjoint(case, seed)
    if kind == "recross":
        wl = W.ch4h_config(ntraj=case["ntraj"], nbeads=case["nbeads"])
        T, P, dt = wl.ntraj, wl.nbeads, wl.dt_au
        q0 = start_geometry(case, seed)
        par = np.repeat(q0[None], P, axis=0) + np.random.default_rng(seed + 1).normal(0.0, JITTER, (P,) + q0.shape)
        traj, bead = np.meshgrid(np.arange(T), np.arange(P), indexing="ij")
        z = normals(seed & 0xFFFFFFFF, traj & ~1, bead, 0, 5, q0.size).reshape((T, P) + q0.shape)
        m = _t(wl.mass)
        p = _t(z * np.where(np.arange(T) % 2, -1.0, 1.0)[:, None, None, None]) * torch.sqrt(m * P / wl.beta)[:, None]
        q = _t(par).expand(T, *par.shape).clone()
        force = lambda x: surface("ch4h")(x)[1]  # noqa: E731
        K, f = ring_map(P, wl.beta, dt), force(q)
        for _ in range(case["steps"]):
            q, p, f = step(q, p, f, m, K, dt, force, False)
        return [q, p, f, None, None, None]
    if kind == "umbrella" and case["pes"] == "h3":
        return _exact_umbrella(case, seed)
    if kind == "qmdff" and case["thermostat"] != "pile":
        u = qmdff_input(case, seed)
        E, m, P = QMDFFEnergy(u["ff"]), _t(u["mass"]), case["nbeads"]
        if case["ntraj"] * P * case["steps"] * len(u["ff"].nci) > 1.2e9:
            return None
        force = lambda x: grad_of(E, x)[1]  # noqa: E731
        q, p, K = u["q"], u["p"], ring_map(P, u["beta"], u["dt"])
        f = force(q)
        for _ in range(case["steps"]):
            q, p, f = step(q, p, f, m, K, u["dt"], force, True)
        return [q, p, f]
    return None  # noise in every step, the barostat's virial, or a surface of several hundred lines


def _exact_umbrella(case, seed):
    u = umbrella_input(case, seed)
    m, P, beta, me = _t(u["mass"]), case["nbeads"], u["beta"], u["mech"]
    xt = _t(u["centers"])

    def xi_of(c):
        bond = lambda ab: (c[:, ab[0] - 1] - c[:, ab[1] - 1]).norm(dim=-1)  # noqa: E731
        com = lambda at: (c[:, [k - 1 for k in at]] * m[[k - 1 for k in at], None]).sum(1) / m[[k - 1 for k in at]].sum()  # noqa: E731,E501
        s1 = (bond(me["bond_break"]) - me["break_ref"]) - (bond(me["bond_form"]) - me["form_ref"])
        s0 = me["r_inf"] - (com(me["reac2"]) - com(me["reac1"])).norm(dim=-1)
        return s0 / (s0 - s1)

    seen = []

    def force(q):
        r = grad_of(h3_energy, q)
        if r is None:
            return None
        c = q.mean(1).detach().requires_grad_(True)
        xi = xi_of(c)
        d = torch.autograd.grad(xi.sum(), c, create_graph=True)[0]
        fs2 = (d * d / m[:, None]).sum((1, 2)) / (2.0 * math.pi * beta)
        bias = 0.5 * u["kforce"] * (xi - xt) ** 2 - 0.5 * torch.log(fs2) / beta
        seen.append(xi.detach())
        return r[1] + torch.autograd.grad(bias.sum(), c)[0][:, None]

    q, p, K = _t(u["q"]), _t(u["p"]), ring_map(P, beta, u["dt"])
    r = grad_of(h3_energy, q)  # set_state's forces are the surface's alone
    if r is None:
        return None
    f = r[1]
    for _ in range(case["steps"]):
        r = step(q, p, f, m, K, u["dt"], force, True)
        if r is None:
            return None
        q, p, f = r
    if case["precision"] == "mixed":
        return [q, p, f]
    x = torch.stack(seen)
    return [q, p, f, x.sum(0), (x * x).sum(0), None]


def _exact_adjoint(case, seed):
    u = qmdff_input(case, seed)
    ff, m, P, dt = u["ff"], _t(u["mass"]), case["nbeads"], u["dt"]
    E = QMDFFEnergy(ff)
    cut, i, j = E.cut[2], *E.nci.T
    base = E.theta
    qq = (E.e1 * base[cut:][i] * base[cut:][j]).detach()
    th = torch.cat([base[:cut], qq]).requires_grad_(True)

    def energy(x):
        r = (x[:, i] - x[:, j]).norm(dim=-1)
        full = E(x, torch.cat([th[:cut], torch.zeros_like(base[cut:])]))
        return full + torch.where(r <= 50.0, th[cut:] / r, torch.zeros_like(r)).sum(-1)

    def force(q):
        x = q.reshape(-1, *q.shape[-2:])
        return torch.autograd.grad(energy(x).sum(), x, create_graph=True)[0].reshape(q.shape)

    q0, p0 = u["q"].clone().requires_grad_(True), u["p"].clone().requires_grad_(True)
    K = ring_map(P, u["beta"], dt)
    # reverse mode one step at a time: the states forward, then each step's vector-Jacobian product
    states = [(q0.detach(), p0.detach())]
    for _ in range(case["steps"]):
        q, p = (x.requires_grad_(True) for x in (states[-1][0].clone(), states[-1][1].clone()))
        q1, p1, _ = step(q, p, force(q), m, K, dt, force, False)
        states.append((q1.detach(), p1.detach()))
    qk, pk = states[-1]
    lq, lp, grad = qk - states[0][0], pk * 1e-3, torch.zeros_like(th)
    for q, p in reversed(states[:-1]):
        q, p = q.clone().requires_grad_(True), p.clone().requires_grad_(True)
        q1, p1, _ = step(q, p, force(q), m, K, dt, force, False)
        lq, lp, g = torch.autograd.grad((q1 * lq).sum() + (p1 * lp).sum(), (q, p, th))
        grad = grad + g
    return [qk, pk, grad, lq, lp]
