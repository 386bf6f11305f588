"""The work that a user of this framework has it do, as measurable cases.

A case is a dict of plain values; `prepare` makes the simulation and its
initial fields on the GPU, `run` takes one pass through the public entry points
(mpulse_b200.runtime.Simulation, mpulse_b200.adjoint), `work` counts the bytes
and operations the pass cannot do without, and `exact` is the same pass in
plain torch in 64 bits (the scheme written out on whole arrays, independent of
the library).

Units and media are those of mpulse_b200.configs: c = 1, lengths in um,
dx = 40 nm, the two-pole silica-like medium, the 800 nm carrier.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mpulse_b200 import abi, adjoint, runtime

DX = 0.04                     # cell size, um (mpulse_b200.configs)
COURANT = 0.45                # stable with the two-pole medium
K0 = 2 * math.pi / 0.8        # 800 nm carrier
SILICA = ((0.6961663, 0.0684), (0.4079426, 0.1162))  # (Delta eps, resonance in um)
ONE_POLE = ((0.5, 0.1),)
FIELDS = ("Ex", "Ey", "Ez", "Bx", "By", "Bz")
NAMES = {"eps": "DesignEps", "chi": "DesignChiScale"}


# ---------------------------------------------------------------------------
# The cases


def listed():
    return [
        # MPulse's driver with this solver plugged in advances one step per
        # call, on the default configuration: 32^3, periodic, FP64
        dict(name="one_step_32_fp64", what="step", nx=32, ny=32, nz=32, bits=64, solver="lin", poles=0, cpml="none",
             d=0, periodic=True, source="none", plasma=False, steps=1),
        # the vacuum pulse workload
        dict(name="vacuum_64_fp32", what="step", nx=64, ny=64, nz=64, bits=32, solver="lin", poles=0, cpml="z", d=8,
             periodic=False, source="none", plasma=False, steps=50),
        # the linear dispersive workload, vacuum in front of the medium
        dict(name="dispersive_128_fp32", what="step", nx=128, ny=128, nz=128, bits=32, solver="lin", poles=2,
             cpml="z", d=10, periodic=False, source="gauss", plasma=False, steps=20),
        # the headline workload: dispersion, Kerr, CPML on all faces, focused
        # pulse; both precisions
        dict(name="kerr_256x256x512_fp32", what="step", nx=256, ny=256, nz=512, bits=32, solver="kerr", poles=2,
             cpml="all", d=12, periodic=False, source="short", plasma=False, steps=10),
        dict(name="kerr_192x192x384_fp64", what="step", nx=192, ny=192, nz=384, bits=64, solver="kerr", poles=2,
             cpml="all", d=12, periodic=False, source="short", plasma=False, steps=5),
        # MPulse's plain and simple-nonlinear solvers, on grids of no round size
        dict(name="plain_150x131x210_fp32", what="step", nx=150, ny=131, nz=210, bits=32, solver="plain", poles=0,
             cpml="none", d=0, periodic=True, source="none", plasma=False, steps=20),
        dict(name="nl_101x75x163_fp64", what="step", nx=101, ny=75, nz=163, bits=64, solver="nl", poles=0,
             cpml="none", d=0, periodic=False, source="none", plasma=False, steps=10),
        # the plasma plug-ins in a Kerr medium
        dict(name="plasma_128x128x192_fp32", what="step", nx=128, ny=128, nz=192, bits=32, solver="kerr", poles=2,
             cpml="all", d=10, periodic=False, source="gauss", plasma=True, steps=10),
        # a trial point of an optimiser's line search: the objective alone,
        # the flux through a plane behind the medium
        dict(name="objective_128x128x256_fp32", what="objective", nx=128, ny=128, nz=256, bits=32, solver="kerr",
             poles=2, cpml="all", d=10, periodic=False, source="short", plasma=False, steps=40, objective="sz",
             every=0, budget=0.0),
        # an optimiser's iteration through torch.autograd: the 96^3 workload
        dict(name="gradient_96_fp32", what="gradient", nx=96, ny=96, nz=96, bits=32, solver="lin", poles=1,
             cpml="all", d=10, periodic=False, source="gauss", plasma=False, steps=300, objective="e2", every=50,
             budget=0.0),
        # a crop of the large nonlinear adjoint in FP64, checkpoints under a
        # memory budget
        dict(name="adjoint_120x104x136_fp64", what="adjoint", nx=120, ny=104, nz=136, bits=64, solver="kerr", poles=2,
             cpml="all", d=8, periodic=False, source="short", plasma=False, steps=60, objective="sz", every=0,
             budget=6e9),
        # a run under observation: energy, the pulse's position and a field to
        # the host every few steps
        dict(name="watched_160x144x250_fp32", what="watch", nx=160, ny=144, nz=250, bits=32, solver="lin", poles=1,
             cpml="z", d=10, periodic=False, source="gauss", plasma=False, steps=10),
    ]


def draw(rng):
    """One more case of the same ranges."""
    what = rng.choices(("step", "objective", "gradient", "adjoint", "watch"), (11, 2, 2, 2, 3))[0]
    design = what in ("gradient", "adjoint")
    bits = rng.choice((32, 32, 64))
    most = (0.9e6 if design else 2.4e7) * (1 if bits == 32 else 0.5)
    while True:
        low, high = (32, 128) if design else (24, 400)
        n = [int(round(math.exp(rng.uniform(math.log(low), math.log(high))))) for _ in range(3)]
        if rng.random() < 0.4:  # users like round sizes
            n = [max(32, (v + 16) // 32 * 32) for v in n]
        cells = n[0] * n[1] * n[2]
        if cells <= most:
            break
    if design:
        solver = rng.choice(("lin", "kerr"))
    elif what == "step":
        solver = rng.choice(("plain", "nl", "lin", "lin", "kerr", "kerr"))
    else:
        solver = rng.choice(("lin", "kerr"))
    plrc = solver in ("lin", "kerr")
    cpml = rng.choice(("z", "all", "all") if not design and plrc else ("all",)) if plrc else "none"
    periodic = not plrc and rng.random() < 0.5
    upto = (1.2e8 if design else 2.4e8) * (1 if bits == 32 else 0.5)
    steps = int(max(1, min(upto / cells, math.exp(rng.uniform(0, math.log(100))))))
    if design:
        steps = int(max(10, min(upto / cells, rng.uniform(20, 200))))
    case = dict(what=what, nx=n[0], ny=n[1], nz=n[2], bits=bits, solver=solver,
                poles=(rng.choice((1, 2)) if design else rng.choice((0, 1, 2, 2))) if plrc else 0, cpml=cpml,
                d=rng.choice((6, 8, 10)) if cpml != "none" else 0, periodic=periodic,
                source=rng.choice(("gauss", "short")) if plrc else "none",
                plasma=plrc and what == "step" and rng.random() < 0.2, steps=steps)
    if what in ("objective", "gradient", "adjoint"):
        case["objective"] = rng.choice(("e2", "sz"))
        case["every"] = rng.choice((0, 25, 50)) if what != "objective" else 0
        case["budget"] = float(rng.choice((0, 8e9))) if what != "objective" and not case["every"] else 0.0
    return case


# ---------------------------------------------------------------------------
# What a case means, in numbers


def numbers(case):
    """The physical parameters of a case."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    d = case["d"]
    q = dict(nx=nx, ny=ny, nz=nz, dx=DX, dt=COURANT * DX, eps=1.5 if case["solver"] == "nl" else 1.0,
             chi=0.05 if case["solver"] == "nl" else 0.02 if case["solver"] == "kerr" else 0.0)
    q["poles"] = []
    for de, lam in (() if not case["poles"] else ONE_POLE if case["poles"] == 1 else SILICA):
        om = 2 * math.pi / lam
        q["poles"].append((de, 0.5e-3 * om, om * om))  # eps, delta, om2
    # the medium starts behind the injection plane, at an eighth of the grid
    q["distance"] = min(nz - 2, d + 6)
    q["z0"] = max(q["distance"] + 4, nz // 8) if case["source"] != "none" and case["poles"] else 0
    q["z1"] = nz + 1
    q["sigma"] = -4 * math.log(1e-6) / (2 * d * DX) if d else 0.0
    if case["source"] == "gauss":  # 10 fs plane pulse along z
        width = K0 * 0.299792458 * 10.0 / math.sqrt(2 * math.log(2))
        q["width"], q["offset"] = width, 3.0 * width
        q["time"] = int((2.5 * width) / (K0 * q["dt"]))  # shortly before its peak
    elif case["source"] == "short":  # 20 fs pulse focused into the medium, waist 2 um
        q["length"] = 0.299792458 * 20.0 / math.sqrt(2 * math.log(2))
        q["waist"] = 2.0
        centre = 0.5 * (nz + 1)
        q["zshift"] = (nz * 0.4 - centre) * DX
        q["tshift"] = 3.0 * q["length"] - ((q["distance"] - centre) * DX - q["zshift"])
        q["time"] = int(2.5 * q["length"] / q["dt"])
    else:
        q["time"] = 0
    if case["plasma"]:
        q |= dict(nu=0.01, mpa=0.02, wion=0.5, K=3, em=0.5, gamma=0.1, rho_bg=0.02)
    if case["what"] in ("gradient", "adjoint"):  # a third of the grid in each direction
        q["design"] = tuple(v for n, lo in ((nx, 1), (ny, 1), (nz, max(q["z0"], 1)))
                            for v in (max(lo, n // 3 + 1), min(n, max(lo, n // 3 + 1) + n // 3 - 1)))
    if "objective" in case:
        z = nz - d - 4
        q["box"] = (nx // 2 - 3, nx // 2 + 4, ny // 2 - 3, ny // 2 + 4, z - 7, z) if case["objective"] == "e2" \
            else (1, nx, 1, ny, z, z)
    return q


def config(case):
    q = numbers(case)
    c = abi.default_config()
    c.nx, c.ny, c.nz = q["nx"], q["ny"], q["nz"]
    c.dx = c.dy = c.dz = q["dx"]
    c.dt, c.eps, c.chi = q["dt"], q["eps"], q["chi"]
    c.precision = abi.MP_FP32 if case["bits"] == 32 else abi.MP_FP64
    c.solver = {"plain": abi.MP_SOLVER_PLAIN, "nl": abi.MP_SOLVER_NL, "lin": abi.MP_SOLVER_PLRC_LIN,
                "kerr": abi.MP_SOLVER_PLRC_NONLIN}[case["solver"]]
    c.boundary = abi.MP_BOUNDARY_PERIODIC if case["periodic"] else abi.MP_BOUNDARY_XY_PERIODIC
    for n in range(abi.MP_MAX_POLES):
        c.poles[n].eps, c.poles[n].delta, c.poles[n].om2 = q["poles"][n] if n < len(q["poles"]) else (0.0, 0.0, 1.0)
    c.medium_z0, c.medium_z1 = q["z0"], q["z1"]
    c.cpml = {"none": abi.MP_CPML_NONE, "z": abi.MP_CPML_Z, "all": abi.MP_CPML_ALL}[case["cpml"]]
    if case["d"]:
        c.cpml_d, c.cpml_kappa_max, c.cpml_a_max, c.cpml_sigma_max = case["d"], 1.0, 0.0, q["sigma"]
    if case["source"] != "none":
        c.n_sources = 1
        s = c.sources[0]
        s.distance, s.eps = q["distance"], 1.0
        if case["source"] == "gauss":
            s.kind = abi.MP_SOURCE_PLANE_GAUSS
            s.k[:], s.H[:] = (0.0, 0.0, K0), (0.0, 1.0, 0.0)
            s.width, s.offset = q["width"], q["offset"]
        else:
            s.kind = abi.MP_SOURCE_SHORT_PULSE
            s.length, s.waist, s.om0, s.amp = q["length"], q["waist"], K0, 1.0
            s.t_shift, s.z_shift = q["tshift"], q["zshift"]
    if case["plasma"]:
        c.plasma, c.plasma_current = 1, 1
        c.plasma_nu, c.plasma_mpa, c.plasma_wion, c.plasma_k = q["nu"], q["mpa"], q["wion"], q["K"]
        c.plasma_em, c.plasma_gamma, c.plasma_rho_bg = q["em"], q["gamma"], q["rho_bg"]
    if "design" in q:
        c.design_box[:] = q["design"]
    return c


def dtype_of(case):
    return torch.float32 if case["bits"] == 32 else torch.float64


def initial(case, seed):
    """The six fields at the start: a few waves of 12 to 40 cells' length under
    a broad envelope, on the planes 0..nz+1 (zero on the walls)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng(seed)
    dev = torch.device("cuda")
    z = torch.arange(nz + 2, device=dev, dtype=torch.float64)[:, None, None]
    y = torch.arange(ny, device=dev, dtype=torch.float64)[None, :, None]
    x = torch.arange(nx, device=dev, dtype=torch.float64)[None, None, :]
    out = {}
    for name in FIELDS:
        f = torch.zeros((nz + 2, ny, nx), device=dev, dtype=torch.float64)
        for _ in range(3):
            kx = 2 * math.pi * r.integers(-2, 3) / nx
            ky = 2 * math.pi * r.integers(-2, 3) / ny
            kz = 2 * math.pi * max(1, round(nz / r.uniform(12, 40))) / nz
            f += r.uniform(0.05, 0.2) * torch.cos(kx * x + ky * y + (kz * z + r.uniform(0, 2 * math.pi)))
        if not case["periodic"]:
            f *= torch.sin(math.pi * z / (nz + 1)) ** 2
            f[0] = f[-1] = 0
        else:
            f[0], f[-1] = f[-2], f[1]
        out[name] = f.to(dtype_of(case))
    return out


def maps(case, seed):
    """The design maps: eps_inf in [1, 4] and, with Kerr, a chi factor in [0.5, 1.5]."""
    q = numbers(case)
    b = q["design"]
    shape = (b[5] - b[4] + 1, b[3] - b[2] + 1, b[1] - b[0] + 1)
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = {"eps": 1.0 + 3.0 * torch.rand(shape, generator=g, device="cuda", dtype=dtype_of(case))}
    if case["solver"] == "kerr":
        out["chi"] = 0.5 + torch.rand(shape, generator=g, device="cuda", dtype=dtype_of(case))
    return out


def objective_of(case):
    kind = abi.MP_OBJ_E2_BOX if case["objective"] == "e2" else abi.MP_OBJ_SZ_PLANE
    return abi.adjoint_config(kind, numbers(case)["box"], case["steps"], checkpoint_every=case["every"],
                              mem_budget=case["budget"])


class DeviceArray:
    """A field of a simulation in place, for torch.as_tensor (keeps the simulation alive)."""

    def __init__(self, sim, name):
        self.sim = sim
        ptr, _, size = sim.device_field(name)
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": sim.cfg.field_shape(),
                                         "typestr": "<f%d" % size, "version": 3}


def view(sim, name):
    return torch.as_tensor(DeviceArray(sim, name), device="cuda")


def simulation(case, seed):
    sim = runtime.Simulation(config(case))
    for name, f in initial(case, seed).items():
        view(sim, name).copy_(f)
    sim.time = numbers(case)["time"]
    return sim


# ---------------------------------------------------------------------------
# One pass


def prepare(case, seed):
    s = {"case": case}
    if case["what"] == "gradient":
        # the optimiser's problem: no initial field, the injected pulse alone,
        # at times that differ with the seed
        s["problem"] = adjoint.DesignProblem(config(case), None, objective_of(case),
                                             start_time=numbers(case)["time"] + seed % 8)
        s["maps"] = {k: m.requires_grad_() for k, m in maps(case, seed).items()}
    else:
        s["sim"] = simulation(case, seed)
        s["fields"] = [view(s["sim"], n) for n in FIELDS]
        if case["periodic"]:  # the ghost planes are images, filled on download only
            s["fields"] = [f[1:-1] for f in s["fields"]]
        if case["plasma"]:
            s["fields"] += [view(s["sim"], n)[1:-1] for n in ("PlasmaDensity", "PlasmaJx", "PlasmaJy", "PlasmaJz")]
        if case["what"] == "adjoint":
            for k, m in maps(case, seed).items():
                s["sim"].upload_design(NAMES[k], m.cpu().numpy())
        if case["what"] != "step" and case["what"] != "watch":
            s["objective"] = objective_of(case)
        if case["what"] == "watch":
            s["host"] = np.empty(case["nx"] * case["ny"] * (case["nz"] + 2))
            s["line"] = (case["nx"] // 2, case["ny"] // 2, 1)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    real = np.float32 if case["bits"] == 32 else np.float64  # the precision the results have
    if case["what"] == "step":
        s["sim"].step(case["steps"])
        return s["fields"]
    if case["what"] == "objective":
        J = s["sim"].objective(s["objective"])
        return [real(J), s["fields"]]
    if case["what"] == "gradient":
        m = s["maps"]
        J = adjoint.design_objective(s["problem"], m["eps"], None, m.get("chi"))
        return [J.detach(), list(torch.autograd.grad(J, list(m.values())))]
    if case["what"] == "adjoint":
        J, g = s["sim"].adjoint(s["objective"])
        return [real(J), [g[NAMES[k]].astype(real) for k in (("eps", "chi") if case["solver"] == "kerr" else ("eps",))],
                s["fields"]]
    sim = s["sim"]  # watch
    sim.step(case["steps"])
    energy = sim.field_energy()
    _, position = sim.follow_max("Ex", 2, s["line"], case["nz"] // 2)
    seen = torch.from_numpy(sim.download("Ex", s["host"])).to(dtype_of(case))
    return [real(energy), real(position), seen, s["fields"]]


def work(case):
    """Per step: each field, accumulator, CPML layer and plasma array read once
    and written once; the reverse steps of an adjoint do the same for the
    adjoint state and read E before and after the step."""
    q = numbers(case)
    nx, ny, nz = q["nx"], q["ny"], q["nz"]
    N, size = nx * ny * nz, case["bits"] // 8
    med = nx * ny * (nz - max(q["z0"], 1) + 1) if case["poles"] else 0
    layers = {"none": 0, "z": 2 * case["d"] * nx * ny,
              "all": 2 * case["d"] * (nx * ny + nx * nz + ny * nz)}[case["cpml"]]
    values = 12 * N + 12 * case["poles"] * med + 8 * layers + (8 * N if case["plasma"] else 0)
    ops = 48 * N + 42 * case["poles"] * med + 12 * layers
    if case["solver"] in ("kerr", "nl"):
        ops += 40 * N
    steps, more = case["steps"], 0
    if case["what"] in ("gradient", "adjoint"):
        values, ops = 2 * values + 6 * N, 2 * ops
    if case["what"] == "watch":
        more = 6 * N * size + 8 * nx * ny * (nz + 2)
    return {"bytes": float(steps * values * size + more), "flops": float(steps * ops)}


# ---------------------------------------------------------------------------
# The same in 64 bits, on whole arrays in torch


def faddeeva(z):
    """w(z) for Im z >= 0, Weideman, SIAM J. Numer. Anal. 31 (1994) 1497-1518."""
    N = 48
    L = math.sqrt(N / math.sqrt(2.0))
    m = np.arange(-2 * N + 1, 2 * N)
    t = L * np.tan(m * math.pi / (4 * N))
    f = np.concatenate([[0.0], np.exp(-t * t) * (L * L + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (4 * N)
    Z = (L + 1j * z) / (L - 1j * z)
    p = torch.zeros_like(z)
    for c in a[N:0:-1]:
        p = p * Z + float(c)
    return 2 * p / (L - 1j * z) ** 2 + (1 / math.sqrt(math.pi)) / (L - 1j * z)


def with_faddeeva(s0, tau, T, tb, B, C, D):
    """B e^{-tb^2} + C e^{-tb^2} w(an) - D e^{-tb^2} w(ap), an = -i tb + tau / T, ap = i tb + tau / T,
    by the reflection w(-z) = 2 e^{-z^2} - w(z) where the argument lies below."""
    total = B * s0
    for sign, c, side in ((-1, C, 1), (1, D, -1)):
        a = sign * 1j * tb + tau / T
        low = a.imag < 0
        w = s0 * faddeeva(torch.where(low, -a, a))
        e = 2 * torch.exp(-2j * sign * tau * tb / T - tau * tau / T ** 2)
        total = total + side * c * torch.where(low, e - w, w)
    return total


def short_pulse(q, which, x, y, z, t):
    """The fields of the focused short pulse of duration T at (x, y, z, t):
    'e' the electric field, 'bx' / 'by' the magnetic ones, unnormalised, phase 0."""
    T, Zr = q["length"], 0.5 * K0 * q["waist"] ** 2
    tb, s0 = 0.5 * K0 * T, math.exp(-(0.5 * K0 * T) ** 2)
    r2 = x * x + y * y
    beam = torch.complex(torch.as_tensor(z, dtype=torch.float64, device=r2.device).expand_as(r2),
                         torch.full_like(r2, Zr))
    R = Zr / beam
    Rp = -Zr / beam ** 2
    tau = (t - z) - r2 / (2 * beam)
    root = math.sqrt(math.pi) * R
    plus, minus = T * tb + 1j * tau, T * tb - 1j * tau
    common = -2j * T + 4j * tau  # T (-i - 2 tb - i + 2 tb) + 4 i tau
    if which == "e":
        tz = -1 - r2 / (2 * beam ** 2)
        B = R * T * (2j * Rp * T ** 2 - R * common * tz)
        C = 1j * root * plus * (Rp * T ** 2 + 2j * R * T * tb * tz - 2 * R * tau * tz)
        D = root * minus * (1j * Rp * T ** 2 + 2 * R * minus * tz)
        return (-1j * with_faddeeva(s0, tau, T, tb, B, C, D) / (root * T ** 4)).real
    scale = math.sqrt(math.pi) * T ** 4
    tx, ty = -x / beam, -y / beam
    if which == "bx":
        B, C, D = -tx * ty * R * T * common, -2 * tx * ty * root * plus ** 2, -2 * tx * ty * root * minus ** 2
        return (1j * with_faddeeva(s0, tau, T, tb, B, C, D) / scale).real
    tz = -1 + r2 / (2 * beam ** 2)
    txx, tzz = -1 / beam, -r2 / beam ** 3
    Rpp = 2 * Zr / beam ** 3
    B = -tx ** 2 * R * T * common + 2j * T ** 2 * txx * R * T
    C = -2 * tx ** 2 * root * plus ** 2 + 1j * T ** 2 * txx * root * plus
    D = -2 * tx ** 2 * root * minus ** 2 + 1j * T ** 2 * txx * root * (-minus)
    first = with_faddeeva(s0, tau, T, tb, B, C, D) / scale
    B = 2 * T * (4j * Rp * T ** 2 * tz - R * ((-2j * T) * tz ** 2 + 2j * (2 * tau * tz ** 2 - T ** 2 * tzz)))
    C = root * (Rpp * R * T ** 4 + 2j * R * plus * (2 * Rp * T ** 2 * tz + R * (
        2j * T * tb * tz ** 2 - 2 * tau * tz ** 2 + T ** 2 * tzz))) / R ** 2
    D = root * (Rpp * R * T ** 4 - 2 * R * minus * (2j * Rp * T ** 2 * tz + R * (
        2 * T * tb * tz ** 2 - 2j * tau * tz ** 2 + 1j * T ** 2 * tzz))) / R ** 2
    second = with_faddeeva(s0, tau, T, tb, B, C, D) / (2 * scale)
    return (1j * (second - first)).real


class Scheme:
    """The time step on whole arrays [nz + 2, ny, nx], 64 bits, differentiable."""

    def __init__(self, case, design=None):
        self.case, self.q = case, numbers(case)
        q = self.q
        self.dev = torch.device("cuda")
        nx, ny, nz = self.n = (q["nx"], q["ny"], q["nz"])
        d, dt = case["d"], q["dt"]
        self.plrc = case["solver"] in ("lin", "kerr")
        self.klo = 1 if case["periodic"] else 0
        self.ehi = nz + 1 if not self.plrc and not case["periodic"] else nz
        # CPML: b and c / dx along each axis (kappa = 1, a = 0), E and H side
        self.layers = []
        for axis, n in ((1, ny), (0, nx), (2, nz)):
            if case["cpml"] == "none" or (case["cpml"] == "z" and axis != 2):
                continue
            for side in "EH":
                b, c = np.zeros(n + 2), np.zeros(n + 2)
                for low in (True, False):
                    far = 0 if side == "H" and low else 1
                    for k in range(d):
                        x = 1 - (k - (0.5 if side == "H" else 0.0)) / d
                        sigma = x ** 3 * q["sigma"]
                        at = far + k if low else n + 1 - far - k
                        b[at] = math.exp(-sigma * dt)
                        c[at] = (b[at] - 1) / DX if sigma else 0.0
                if axis == 2:
                    if case["periodic"] and side == "H":
                        b[0] = c[0] = 0
                    shape = (n + 2, 1, 1)
                else:
                    b, c, shape = b[1:-1], c[1:-1], (1, n, 1) if axis == 1 else (1, 1, n)
                self.layers.append((side, axis, torch.tensor(b, device=self.dev).reshape(shape),
                                    torch.tensor(c, device=self.dev).reshape(shape)))
        chi0 = xi0 = 0
        self.poles = []
        for de, delta, om2 in q["poles"]:
            beta = math.sqrt(om2 - delta * delta)
            ph = delta - 1j * beta
            C = complex(np.exp(-ph * dt))
            gam = de * om2 / beta
            a = 1j * gam * (C - 1) / ph
            x = 1j * gam * (C * (ph * dt + 1) - 1) / (ph * ph * dt)
            chi0, xi0 = chi0 + a, xi0 + x
            self.poles.append(((a - x) * (1 - C), x * (1 - C), C))
        chi0, xi0 = complex(chi0).real, complex(xi0).real
        eps, chi = q["eps"], q["chi"]
        if design is not None:
            b = q["design"]
            inside = (slice(b[4], b[5] + 1), slice(b[2] - 1, b[3]), slice(b[0] - 1, b[1]))
            whole = torch.zeros((nz + 2, ny, nx), device=self.dev, dtype=torch.float64)

            def placed(m, other):
                return torch.index_put(whole + other, tuple(torch.meshgrid(*(
                    torch.arange(s.start, s.stop, device=self.dev) for s in inside), indexing="ij")), m)

            eps = placed(design["eps"], eps)
            chi = chi * placed(design["chi"], 1.0) if "chi" in design else chi
        if self.plrc:
            z = torch.arange(nz + 2, device=self.dev).reshape(-1, 1, 1)
            self.medium = (z >= max(q["z0"], 1)) & (z <= min(q["z1"], nz))
            one = torch.ones((), device=self.dev, dtype=torch.float64)
            self.numer = torch.where(self.medium, eps - xi0, one)
            self.denom = torch.where(self.medium, eps + chi0 - xi0, one)
            self.chi = torch.where(self.medium, chi * one, 0 * one)
        self.planes = {}

    def start(self, fields):
        """The state: E, B, the accumulators, the layers, the plasma."""
        E, B = [fields[n].double() for n in FIELDS[:3]], [fields[n].double() for n in FIELDS[3:]]
        zero = lambda: torch.zeros_like(E[0])  # noqa: E731
        return E + B + [zero() for _ in range(6 * len(self.poles) + 2 * len(self.layers) + 4 * self.case["plasma"])]

    def source(self, side, t):
        """The two injected components (x, y) on the plane, per dx."""
        q, l = self.q, self.q["distance"] - 1
        i = torch.arange(1, self.n[0] + 1, device=self.dev, dtype=torch.float64)[None, :]
        j = torch.arange(1, self.n[1] + 1, device=self.dev, dtype=torch.float64)[:, None]
        ones = torch.ones_like(i + j)
        if self.case["source"] == "gauss":
            if side == "E":  # H at half steps: Hy = 1
                pos = K0 * (l + 0.5) * DX + K0 * q["dt"] * (t - 0.5)
            else:            # E: Ex = k x H, opposite sign
                pos = K0 * l * DX + K0 * q["dt"] * t
            a = (pos - q["offset"]) / q["width"]
            v = math.exp(-a * a) * math.sin(pos)
            return (v * ones / DX, 0 * ones) if side == "E" else (0 * ones, v * ones / DX)
        cx, cy, cz = (0.5 * (n + 1) for n in self.n)
        xo, xh, yo, yh = (i - cx) * DX * ones, (i + 0.5 - cx) * DX * ones, (j - cy) * DX * ones, (j + 0.5 - cy) * DX * ones
        if "peak" not in self.planes:
            zero = torch.zeros((1, 1), device=self.dev, dtype=torch.float64)
            self.planes["peak"] = float(short_pulse(q, "e", zero, zero, 0.0, 0.0))
        peak = self.planes["peak"]
        if side == "H":
            e = short_pulse(q, "e", xh, yo, (l - cz) * DX - q["zshift"], t * q["dt"] - q["tshift"])
            return 0 * ones, e / peak / DX
        z, s = (l - 0.5 - cz) * DX - q["zshift"], (t - 0.5) * q["dt"] - q["tshift"]
        return short_pulse(q, "by", xh, yo, z, s) / peak / DX, short_pulse(q, "bx", xo, yh, z, s) / peak / DX

    def added(self, J, side, t):
        if self.case["source"] == "none":
            return J
        at = self.q["distance"] - (side == "H")
        if (side, t) not in self.planes:
            self.planes[side, t] = self.source(side, t)
        a, b = self.planes[side, t]
        pick = torch.zeros((self.n[2] + 2, 1, 1), device=self.dev, dtype=torch.float64)
        pick[at] = 1.0
        return [J[0] + pick * a, J[1] + pick * b, J[2]]

    def up(self, f, axis):
        """f at the next index along the axis (planes beyond the last: see below)."""
        if axis != 2:
            return torch.roll(f, -1, 2 - axis)
        last = f[1:2] if self.case["periodic"] else f[-1:]
        return torch.cat([f[1:-1], last, f[-1:]]) if self.case["periodic"] else torch.cat([f[1:], last])

    def down(self, f, axis):
        if axis != 2:
            return torch.roll(f, 1, 2 - axis)
        first = f[-2:-1] if self.case["periodic"] else f[:1]
        return torch.cat([f[:1], first, f[1:-1]]) if self.case["periodic"] else torch.cat([f[:1], f[:-1]])

    def curl(self, F, shift, sign):
        """The differences sign * (F - shifted F) per axis, of all components."""
        return [[sign * (F[c] - shift(F[c], a)) if c != a else None for c in range(3)] for a in range(3)]

    def currents(self, side, D, psi):
        """The layers' currents from the differences; returns (J, new psi)."""
        J, new, at = [0.0, 0.0, 0.0], [], 0
        own = [l for l in self.layers if l[0] == side]
        s = -1.0 if side == "E" else 1.0
        for (_, axis, b, c), p in zip(own, zip(psi[::2], psi[1::2])):
            # axis a feeds the next two components u, v: differences of v, u
            u, v = (axis + 1) % 3, (axis + 2) % 3
            p0 = b * p[0] + c * (s * D[axis][v])
            p1 = b * p[1] + c * (-s * D[axis][u])
            J[u], J[v] = J[u] + p0, J[v] + p1
            new += [p0, p1]
        return J, new

    def rows(self, new, old, lo, hi):
        return torch.cat([old[:lo], new[lo:hi + 1], old[hi + 1:]])

    def step(self, t, *state):
        case, q, dt, nz = self.case, self.q, self.q["dt"], self.n[2]
        state = list(state)
        E, B, rest = state[:3], state[3:6], state[6:]
        psi, rest = rest[:6 * len(self.poles)], rest[6 * len(self.poles):]
        half = len(self.layers)  # two per layer and side, sides alternate
        layE = [x for n, l in enumerate(self.layers) if l[0] == "E" for x in rest[2 * n:2 * n + 2]]
        layH = [x for n, l in enumerate(self.layers) if l[0] == "H" for x in rest[2 * n:2 * n + 2]]
        plasma = rest[2 * half:]
        # ---- E
        D = self.curl(B, self.down, 1.0)
        J, layE = self.currents("E", D, layE)
        J = self.added(J, "E", t)
        curl = [(D[(c + 1) % 3][(c + 2) % 3] - D[(c + 2) % 3][(c + 1) % 3]) / DX for c in range(3)]
        E2 = E[0] ** 2 + E[1] ** 2 + E[2] ** 2
        if case["plasma"]:
            rho, n, m = plasma[0], 0.5 * dt * q["nu"], dt * q["mpa"]
            rho = (rho * (1 + n * E2) + m * E2 ** q["K"]) / (1 - n * E2)
            sig = 0.5 * dt * q["mpa"] * q["wion"] * E2 ** (q["K"] - 1)
            cur = [(plasma[1 + c] * (1 - 0.5 * q["gamma"] * dt) - q["em"] * dt * E[c] * (rho + q["rho_bg"])) /
                   (1 + 0.5 * q["gamma"] * dt) for c in range(3)]
            J = [J[c] + cur[c] for c in range(3)]
            plasma = [self.rows(x, o, 1, nz) for x, o in zip([rho] + cur, plasma)]
        else:
            sig = 0.0
        if case["solver"] == "plain":
            X, A = [E[c] + dt * curl[c] for c in range(3)], None
        elif case["solver"] == "nl":
            X = [((q["eps"] + q["chi"] * E2) * E[c] + dt * curl[c]) / q["eps"] for c in range(3)]
            A = q["chi"] / q["eps"]
        else:
            P, new = [0.0, 0.0, 0.0], []
            for n, (dD, dx, C) in enumerate(self.poles):
                for c in range(3):
                    re, im = psi[6 * n + 2 * c], psi[6 * n + 2 * c + 1]
                    a, b = dD.real * E[c] + re, dD.imag * E[c] + im
                    P[c] = P[c] + torch.where(self.medium, a, 0 * a)
                    new += [torch.where(self.medium, dx.real * E[c] + C.real * a - C.imag * b, re),
                            torch.where(self.medium, dx.imag * E[c] + C.real * b + C.imag * a, im)]
            psi = new
            kerr = case["solver"] == "kerr"
            front = self.numer - sig + (self.chi * E2 if kerr else 0.0)
            X = [(front * E[c] + dt * (curl[c] + J[c]) + P[c]) / (self.denom + sig) for c in range(3)]
            A = self.chi / (self.denom + sig) if kerr else None
        if A is not None:  # |E| + A |E|^3 = |X|, along X
            c2 = X[0] ** 2 + X[1] ** 2 + X[2] ** 2
            some = c2 > 0
            C = torch.sqrt(torch.where(some, c2, torch.ones_like(c2)))
            with torch.no_grad():
                r = C.detach().clone()
                for _ in range(9):
                    r = (2 * A * r ** 3 + C) / (3 * A * r ** 2 + 1)
            r = (2 * A * r ** 3 + C) / (3 * A * r ** 2 + 1)  # carries the derivative
            X = [torch.where(some, x * (r / C), torch.zeros_like(x)) for x in X]
        E = [self.rows(X[c], E[c], 1, self.ehi) for c in range(3)]
        # ---- B
        D = self.curl(E, self.up, -1.0)
        M, layH = self.currents("H", D, layH)
        M = self.added(M, "H", t)
        B = [self.rows(B[c] + dt * ((D[(c + 2) % 3][(c + 1) % 3] - D[(c + 1) % 3][(c + 2) % 3]) / DX + M[c]), B[c],
                       self.klo, nz) for c in range(3)]
        lay, e, h = [], iter(layE), iter(layH)
        for l in self.layers:
            it = e if l[0] == "E" else h
            lay += [next(it), next(it)]
        return tuple(E + B + psi + lay + plasma)

    def term(self, state):
        """The objective's term of a state."""
        b = self.q["box"]
        at = (slice(b[4], b[5] + 1), slice(b[2] - 1, b[3]), slice(b[0] - 1, b[1]))
        E, B = [f[at] for f in state[:3]], [f[at] for f in state[3:6]]
        if self.case["objective"] == "e2":
            return self.q["dt"] * (E[0] ** 2 + E[1] ** 2 + E[2] ** 2).sum()
        return self.q["dt"] * DX * DX * (E[0] * B[1] - E[1] * B[0]).sum()


def outputs(case, state):
    cut = slice(1, -1) if case["periodic"] else slice(None)
    return [f[cut] for f in state[:6]] + ([f[1:-1] for f in state[-4:]] if case["plasma"] else [])


def exact(case, seed):
    q = numbers(case)
    t0 = q["time"] + (seed % 8 if case["what"] == "gradient" else 0)
    if case["what"] in ("gradient", "adjoint"):
        from torch.utils.checkpoint import checkpoint

        m = {k: v.double().requires_grad_() for k, v in maps(case, seed).items()}
        scheme = Scheme(case, m)
        zero = torch.zeros((q["nz"] + 2, q["ny"], q["nx"]), device="cuda", dtype=torch.float64)
        state = tuple(scheme.start(initial(case, seed) if case["what"] == "adjoint" else {n: zero for n in FIELDS}))
        J = 0.0
        for n in range(case["steps"]):
            scheme.planes = {k: v for k, v in scheme.planes.items() if k == "peak"}
            state = checkpoint(scheme.step, t0 + n, *state, use_reentrant=False, preserve_rng_state=False)
            J = J + scheme.term(state)
        g = list(torch.autograd.grad(J, list(m.values())))
        if case["what"] == "gradient":
            return [J.detach(), g]
        return [np.float64(J.detach().item()), g, [f.detach() for f in outputs(case, state)]]
    with torch.no_grad():
        scheme = Scheme(case)
        state = tuple(scheme.start(initial(case, seed)))
        J = 0.0
        for n in range(case["steps"]):
            scheme.planes = {k: v for k, v in scheme.planes.items() if k == "peak"}
            state = scheme.step(t0 + n, *state)
            if case["what"] == "objective":
                J += float(scheme.term(state))
        out = outputs(case, state)
        if case["what"] == "step":
            return out
        if case["what"] == "objective":
            return [np.float64(J), out]
        energy = np.float64(sum(float((f[1:-1] ** 2).sum()) for f in state[:6])) * DX ** 3
        line = state[0][:, case["ny"] // 2 - 1, case["nx"] // 2 - 1].cpu().numpy()
        n, at = case["nz"], case["nz"] // 2
        while True:  # uphill along the line, then the parabola's vertex
            left, mid, right = line[at - 1 or n], line[at], line[at % n + 1]
            if right > mid:
                at = at % n + 1
            elif left > mid:
                at = at - 1 or n
            else:
                break
        return [energy, at + (left - right) / (2 * (left - 2 * mid + right)), state[0], out]
