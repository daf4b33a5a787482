"""Performance cases: the work a user of this package has it do, as calls of its
public entry points.

    listed()             the cases, dicts of plain values
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call
    run(state)           one pass; returns its outputs
    work(case)           bytes and flops of a pass
    exact(case, seed)    the outputs in 64 bits by plain torch, where there is
                         a short way to them

A pass is what a driver does between two outputs: take the state, advance it
by a number of steps, hand the state back.  Kinds of cases:

    rows      single-material steps on a rectangle, the state coming from and
              going to device tensors (the way the slab decomposition couples
              the solver): FP64, both kernel families
    mesh      single-material steps of a state that stays with the solver,
              then the state on the host (the MIXED form has this way only)
    amr       steps on an adaptive mesh with its flags and refinements, then
              the state on the host
    mm        multi-material run from initial data on the host: mixture
              states, steps, cell states on the host
    transfer  scalar VOF transport: u1 in, the time loop on the device, u1 out
    adjoint   gradient of the probe pressure by the discrete adjoint, on device
              tensors
"""
from __future__ import annotations

import math

import numpy as np
import torch

import zephyr_b200 as Z
from zephyr_b200.adjoint import Adjoint
from zephyr_b200.mmf import CrpMode, DirSplit, Material, MixturePT, MmFluid
from zephyr_b200.slabs import GpuSlabSolver, Slab
from zephyr_b200.transfer import Method, Transfer

DEV = "cuda:0"
BOUND = {"wall": 1, "zoe": 2, "periodic": 3}
FLUX = {"HLL": Z.Fluxes.HLL, "HLLC": Z.Fluxes.HLLC}
GAMMA = 1.4
LIQUID = (4.4, 6.0e8)  # gamma, P0 of the stiffened gas
# centre, radius and density of the bubbles of the adaptive cases
BUBBLES = [(0.25, 0.25, 0.07, 8.0), (0.45, 0.30, 0.06, 4.0), (0.30, 0.50, 0.08, 10.0), (0.55, 0.52, 0.05, 6.0),
           (0.42, 0.70, 0.06, 3.0), (0.62, 0.24, 0.06, 12.0)]


def listed():
    return [
        # The first run of a new user: Riemann2D problem at 256^2, every
        # setting at its default (first order, PARITY kernels, HLLC), 200
        # steps.  Small enough that latency and launches count.
        dict(name="riemann_256_first_order", kind="rows", nx=256, ny=256, steps=200, accuracy=1, scheme="pc",
             kernels="PARITY", flux="HLLC", limiter="MC", eos="ideal", bounds="zoe", data="quadrants"),
        # The smallest calls in earnest: a coarse second-order run, odd sizes,
        # channel walls, as in parameter studies and unit checks.
        dict(name="channel_129x67", kind="rows", nx=129, ny=67, steps=200, accuracy=2, scheme="pc", kernels="FAST",
             flux="HLL", limiter="minmod", eos="ideal", bounds="wall", data="quadrants"),
        # The drop-in form at second order on a ragged mesh: bit-exact kernels,
        # the constructor's limiter.
        dict(name="parity_1031x517_second_order", kind="rows", nx=1031, ny=517, steps=20, accuracy=2, scheme="pc",
             kernels="PARITY", flux="HLLC", limiter="MC", eos="ideal", bounds="zoe", data="quadrants"),
        # The benchmark's mesh, predictor-corrector, FP64.
        dict(name="fourier_2048", kind="rows", nx=2048, ny=2048, steps=20, accuracy=2, scheme="pc", kernels="FAST",
             flux="HLLC", limiter="van Albada", eos="ideal", bounds="periodic", data="fourier"),
        # Heun's scheme at an uneven size, with the stiffened gas.
        dict(name="liquid_1500x1100_heun", kind="rows", nx=1500, ny=1100, steps=20, accuracy=2, scheme="heun",
             kernels="FAST", flux="HLLC", limiter="van Albada", eos="stiffened", bounds="periodic", data="fourier"),
        # The MIXED form over a long horizon: 500 steps, then the state.
        dict(name="fourier_1024_mixed", kind="mesh", nx=1024, ny=1024, steps=500, accuracy=2, scheme="pc",
             precision="MIXED", flux="HLLC", limiter="van Albada", bounds="periodic"),
        # The AMR benchmark's mesh (512^2, three levels), adapted every 10
        # steps by the density-gradient criterion: moving interfaces, as many
        # cells at the end of a pass as at its start.
        dict(name="bubbles_512_3_levels", kind="amr", n0=512, levels=3, adapts=5, kernels="FAST", criterion="gradient",
             limiter="van Albada 1"),
        # The drop-in form on an adaptive mesh with the solver's own flags.
        dict(name="bubbles_200_2_levels_parity", kind="amr", n0=200, levels=2, adapts=5, kernels="PARITY",
             criterion="jumps", limiter="MC"),
        # Shock on a water column, the multi-material benchmark's mesh.
        dict(name="column_1024", kind="mm", n=1024, steps=500, accuracy=1, crp="PLIC", split="NONE"),
        # The same problem at second order and a smaller, odd size.
        dict(name="column_451_second_order", kind="mm", n=451, steps=300, accuracy=2, crp="PLIC", split="NONE"),
        # The transfer problem's loop (VOF, split) over a field of disks.
        dict(name="disks_2048x1434", kind="transfer", nx=2048, ny=1434, steps=50, method="VOF", split=True, disks=64),
        # The adjoint benchmark: 1024^2, 100 Heun steps, checkpoints every 10.
        dict(name="adjoint_1024", kind="adjoint", nx=1024, ny=1024, steps=100, every=10),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rows", "rows", "rows", "mesh", "amr", "amr", "mm", "transfer", "adjoint"])
    if kind in ("rows", "mesh"):
        nx = _log(rng, 48, 2048)
        ny = max(17, int(nx * rng.uniform(0.4, 1.0)))
        # as many steps as about 8e7 cell updates take, 10 to 200
        steps = max(10, min(200, int(8.0e7 / (nx * ny))))
        if kind == "mesh":
            return dict(kind=kind, nx=nx, ny=ny, steps=steps, accuracy=2, scheme=rng.choice(["pc", "heun"]),
                        precision="MIXED", flux="HLLC", limiter="van Albada", bounds="periodic")
        kernels = rng.choice(["PARITY", "FAST", "FAST"])
        accuracy = rng.choice([1, 2, 2])
        data = rng.choice(["quadrants", "fourier"])
        return dict(kind=kind, nx=nx, ny=ny, steps=steps // (4 if kernels == "PARITY" else 1) + 1, accuracy=accuracy,
                    scheme=rng.choice(["pc", "pc", "heun"]), kernels=kernels, flux=rng.choice(["HLLC", "HLLC", "HLL"]),
                    limiter=rng.choice(["MC", "minmod", "van Albada", "van Leer"]),
                    eos=rng.choice(["ideal", "ideal", "stiffened"]),
                    bounds="periodic" if data == "fourier" else rng.choice(["zoe", "wall"]), data=data)
    if kind == "amr":
        kernels = rng.choice(["PARITY", "FAST", "FAST"])
        return dict(kind=kind, n0=_log(rng, 64, 400), levels=rng.choice([1, 2, 3]), adapts=rng.choice([2, 3, 5]),
                    kernels=kernels, criterion="jumps" if kernels == "PARITY" else "gradient",
                    limiter=rng.choice(["MC", "van Albada 1"]))
    if kind == "mm":
        return dict(kind=kind, n=_log(rng, 96, 700), steps=rng.choice([50, 100, 200]), accuracy=rng.choice([1, 1, 2]),
                    crp=rng.choice(["PLIC", "PLIC", "VS", "NONE"]), split=rng.choice(["NONE", "SIMPLE", "STRANG"]))
    if kind == "transfer":
        nx = _log(rng, 128, 2200)
        return dict(kind=kind, nx=nx, ny=int(nx * rng.uniform(0.5, 0.9)), steps=rng.choice([10, 20, 40]),
                    method=rng.choice(["VOF", "VOF", "VOF_CRP", "CRP_SE"]), split=rng.choice([True, True, False]),
                    disks=rng.choice([1, 16, 64]))
    nx = _log(rng, 64, 900)
    return dict(kind="adjoint", nx=nx, ny=max(33, int(nx * rng.uniform(0.5, 1.0))), steps=rng.choice([20, 40, 60]),
                every=rng.choice([5, 10]))


# ---- initial data -----------------------------------------------------------------
def _centres(n):
    return (torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) / n


def _modes(rs, nx, ny):
    """A smooth periodic field of eight modes on the unit square."""
    x, y = _centres(nx)[:, None], _centres(ny)[None, :]
    f = torch.zeros(nx, ny, dtype=torch.float64, device=DEV)
    for m in range(1, 9):
        a, phi, psi = rs.uniform(0.0, 1.0) / 8.0, rs.uniform(0.0, 2 * np.pi), rs.uniform(0.0, 2 * np.pi)
        f += a * torch.sin(2 * np.pi * m * x + phi) * torch.sin(2 * np.pi * m * y + psi)
    return f


def _eos(name):
    return Z.StiffenedGas(*LIQUID) if name == "stiffened" else Z.IdealGas(GAMMA)


def _primitive(case, seed):
    """(rho, u, v, p) on the unit square, (nx, ny) tensors: `fourier`, smooth
    modes around a gas at rest; `quadrants`, the four-quadrant Riemann problem
    with the meeting point and the states moved a little by the seed."""
    rs = np.random.RandomState(seed % (1 << 31))
    nx, ny = case["nx"], case["ny"]
    if case.get("data", "fourier") == "fourier":
        r, u, v, p = (_modes(rs, nx, ny) for _ in range(4))
        r, u, v, p = 1.0 + 0.2 * r, 0.3 * u, 0.3 * v, 1.0 + 0.1 * p
    else:
        q = np.array([[1.5, 0.0, 0.0, 1.5], [0.5323, 1.206, 0.0, 0.3], [0.138, 1.206, 1.206, 0.029],
                      [0.5323, 0.0, 1.206, 0.3]]) * rs.uniform(0.95, 1.05, (4, 4))
        east = (_centres(nx) >= rs.uniform(0.4, 0.6))[:, None]
        north = (_centres(ny) >= rs.uniform(0.4, 0.6))[None, :]
        r, u, v, p = (torch.where(north, torch.where(east, q[0, k], q[1, k]), torch.where(east, q[3, k], q[2, k]))
                      .to(torch.float64) for k in range(4))
    if case.get("eos") == "stiffened":  # a liquid: metres per second, pascals
        r, u, v, p = 1000.0 * r, 100.0 * u, 100.0 * v, 1.0e8 * p
    return r, u, v, p


def _state5(case, seed):
    """The five rows of the solver's state, flat: density, velocity, pressure, energy."""
    r, u, v, p = _primitive(case, seed)
    e = _eos(case.get("eos", "ideal")).energy_rP(r, p)
    return torch.stack([t.expand_as(r).contiguous() for t in (r, u, v, p, e)]).reshape(-1)


def _configure(case):
    def setup(solver):
        solver.set_accuracy(case["accuracy"])
        solver.set_CFL(0.4)
        solver.set_method(FLUX[case["flux"]])
        solver.set_limiter(case["limiter"])
        solver.set_scheme(Z.Scheme.HEUN if case["scheme"] == "heun" else Z.Scheme.PREDICTOR_CORRECTOR)
    return setup


# ---- rows: FP64 steps between device tensors --------------------------------------
def _prepare_rows(case, seed):
    slab = Slab(case["nx"], case["ny"], (0.0, 1.0, 0.0, 1.0), (BOUND[case["bounds"]],) * 4, 1, 0)
    gpu = GpuSlabSolver(slab, _eos(case["eos"]), _configure(case), kernels=Z.Kernels[case["kernels"]], device_rows=True)
    return {"gpu": gpu, "in": _state5(case, seed),
            "wait": torch.zeros(case["nx"] * case["ny"], dtype=torch.int32, device=DEV)}


def _run_rows(case, s):
    gpu = s["gpu"]
    gpu.put_rows(0, s["in"], s["wait"])
    gpu.solver.update(gpu.mesh, steps=case["steps"])
    state, wait = gpu.get_rows(0, case["nx"])
    return {"state": state, "wait": wait, "dt": gpu.dt()}


# ---- mesh: MIXED steps of a resident state ----------------------------------------
def _prepare_mesh(case, seed):
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_boundaries(Z.Boundaries(*(BOUND[case["bounds"]],) * 4))
    gen.set_sizes(case["nx"], case["ny"])
    mesh = Z.EuMesh(gen)
    solver = Z.SmFluid(Z.IdealGas(GAMMA), precision=Z.Precision[case["precision"]], kernels=Z.Kernels.FAST)
    _configure(case)(solver)
    solver.add_types(mesh)
    mesh.set_state(*_state5(case, seed).reshape(5, -1).cpu().numpy())
    return {"mesh": mesh, "solver": solver}


def _run_mesh(case, s):
    s["solver"].update(s["mesh"], steps=case["steps"])
    return {"state": s["mesh"].get_state(), "dt": s["solver"].dt()}


# ---- amr: steps with adaptation ----------------------------------------------------
def _bubbles(mesh, scale):
    """Dense bubbles carried along by a gas in pressure balance, at the mesh's
    cell centres.  `scale` multiplies the velocities (the pressure goes with
    its square): the same density field in other units of time, so that every
    seed adapts the mesh alike and gives outputs of one shape."""
    x, y = mesh.centers()
    r = np.ones_like(x)
    for cx, cy, rad, rho in BUBBLES:
        r[np.hypot(x - cx, y - cy) < rad] = rho
    u, v, p = (np.full_like(x, c) for c in (0.9 * scale, 0.45 * scale, scale * scale))
    mesh.set_state(r, u, v, p, p / ((GAMMA - 1.0) * r))


def _adapt(case, s):
    if case["criterion"] == "gradient":
        s["solver"].set_flags_gradient(s["mesh"], 0.05, 0.01, download=False)
    else:
        s["solver"].set_flags(s["mesh"], download=False)
    s["mesh"].refine()


def _prepare_amr(case, seed):
    rs = np.random.RandomState(seed % (1 << 31))
    gen = Z.Rectangle(0.0, 1.0, 0.0, 1.0)
    gen.set_boundaries(Z.Boundaries(*(BOUND["zoe"],) * 4))
    gen.set_sizes(case["n0"], case["n0"])
    mesh = Z.EuMesh(gen)
    mesh.set_max_level(case["levels"])
    solver = Z.SmFluid(Z.IdealGas(GAMMA), kernels=Z.Kernels[case["kernels"]])
    solver.set_accuracy(2)
    solver.set_CFL(0.4)
    solver.set_limiter(case["limiter"])
    solver.add_types(mesh)
    mesh.set_distributor("slope")
    s = {"mesh": mesh, "solver": solver}
    scale = rs.uniform(0.5, 2.0)
    # the driver's initial loop: flags, refinement, the data again
    for _ in range(case["levels"] + 1):
        _bubbles(mesh, scale)
        _adapt(case, s)
    _bubbles(mesh, scale)
    for _ in range(3):  # until the interfaces have their numerical width
        solver.update(mesh, steps=10)
        _adapt(case, s)
    return s


def _run_amr(case, s):
    for _ in range(case["adapts"]):
        s["solver"].update(s["mesh"], steps=10)
        _adapt(case, s)
    return {"state": s["mesh"].get_state(), "dt": s["solver"].dt()}


# ---- mm: shock on a water column -----------------------------------------------------
def _column(n, rs):
    """Air at rest at 1 bar with a water column, and a shock coming in from the
    left, on a square of 0.1 m: (rho, vx, vy, p, beta) per cell."""
    h = 0.1 / n
    c = (np.arange(n) + 0.5) * h
    x, y = np.repeat(c, n), np.tile(c, n)
    cx, cy, rad = 0.05 + 0.004 * rs.uniform(-1, 1), 0.05 + 0.004 * rs.uniform(-1, 1), rs.uniform(0.008, 0.012)
    d = np.hypot(x - cx, y - cy)
    alpha = (d < rad).astype(np.float64)
    cut = np.where(np.abs(d - rad) < h)[0]
    t = ((np.arange(8) + 0.5) / 8 - 0.5) * h
    alpha[cut] = (np.hypot(x[cut, None, None] + t[None, :, None] - cx, y[cut, None, None] + t[None, None, :] - cy)
                  < rad).mean(axis=(1, 2))
    g, p1, r1, p2 = 1.4, 1.0e5, 1.2, rs.uniform(0.8e6, 1.2e6)
    r2 = r1 * ((g + 1) * p2 + (g - 1) * p1) / ((g - 1) * p2 + (g + 1) * p1)
    u2 = math.sqrt((p2 - p1) * (1 / r1 - 1 / r2))
    behind = x < cx - rad - 0.002
    ra = np.where(behind, r2, r1)
    rho = alpha * 1000.0 + (1 - alpha) * ra
    beta = np.zeros((n * n, 2))
    beta[:, 0] = alpha * 1000.0 / rho
    beta[:, 1] = 1.0 - beta[:, 0]
    beta[alpha >= 1.0] = (1.0, 0.0)
    beta[alpha <= 0.0] = (0.0, 1.0)
    return rho, np.where(behind, u2, 0.0), np.zeros(n * n), np.where(behind, p2, p1), beta


def _prepare_mm(case, seed):
    n = case["n"]
    gen = Z.Rectangle(0.0, 0.1, 0.0, 0.1)
    gen.set_boundaries(Z.Boundaries(BOUND["zoe"], BOUND["zoe"], BOUND["wall"], BOUND["wall"]))
    gen.set_sizes(n, n)
    mesh = Z.EuMesh(gen)
    solver = MmFluid(MixturePT([Material.stiffened("Water"), Material.ideal("Air")]))
    solver.set_CFL(0.4)
    solver.set_accuracy(case["accuracy"])
    if case["crp"] == "NONE":
        solver.set_method(Z.Fluxes.HLLC)
    else:
        solver.set_crp_mode(CrpMode[case["crp"]])
    solver.set_splitting(DirSplit[case["split"]])
    solver.add_types(mesh)
    return {"mesh": mesh, "solver": solver, "in": _column(n, np.random.RandomState(seed % (1 << 31)))}


def _run_mm(case, s):
    s["solver"].make_states(s["mesh"], *s["in"])
    s["solver"].update(s["mesh"], steps=case["steps"])
    return {"cells": s["solver"].states(s["mesh"]), "dt": s["solver"].dt()}


# ---- transfer: VOF transport of disks ---------------------------------------------------
def _prepare_transfer(case, seed):
    rs = np.random.RandomState(seed % (1 << 31))
    nx, ny, height = case["nx"], case["ny"], case["ny"] / case["nx"]
    gen = Z.Rectangle(0.0, 1.0, 0.0, height)
    gen.set_boundaries(Z.Boundaries(*(BOUND["zoe"],) * 4))
    gen.set_sizes(nx, ny)
    # volume fractions from the signed distance to the nearest circle, one
    # cell wide
    x, y = _centres(nx)[:, None], height * _centres(ny)[None, :]
    u1 = torch.zeros(nx, ny, dtype=torch.float64, device=DEV)
    for _ in range(case["disks"]):
        rad = rs.uniform(0.1, 0.15) if case["disks"] == 1 else rs.uniform(0.01, 0.04)
        d = torch.hypot(x - rs.uniform(0.2, 0.8), y - height * rs.uniform(0.2, 0.8)) - rad
        u1 = torch.maximum(u1, torch.clamp(0.5 - d * nx, 0.0, 1.0))
    mesh = Z.EuMesh(gen)
    solver = Transfer()
    solver.set_method(Method[case["method"]])
    solver.set_velocity_translation(0.7, -0.35)
    solver.add_types(mesh)
    return {"mesh": mesh, "solver": solver, "in": u1.reshape(-1).cpu().numpy()}


def _run_transfer(case, s):
    mesh, solver = s["mesh"], s["solver"]
    solver.set_u1(mesh, s["in"])
    solver.update_interface(mesh)
    t = solver.advance(mesh, case["steps"], 0.0, 1.0, splitting=case["split"])
    return {"u1": solver.u1(mesh), "t": t}


# ---- adjoint ---------------------------------------------------------------------------
def _prepare_adjoint(case, seed):
    r, u, v, p = (t.contiguous() for t in _primitive(case, seed))
    h = min(1.0 / case["nx"], 1.0 / case["ny"])
    dt = 0.4 * h / float((torch.hypot(u, v) + torch.sqrt(GAMMA * p / r)).max())
    return {"adj": Adjoint(case["nx"], case["ny"]), "in": (r, u, v, p),
            "prm": Adjoint.params(steps=case["steps"], checkpoint_every=case["every"], gamma=GAMMA, dt=dt),
            "grad": torch.empty_like(r)}


def _run_adjoint(case, s):
    J, dgamma = s["adj"].gradient(s["prm"], *s["in"], s["grad"])
    return {"J": J, "drho": s["grad"], "dgamma": dgamma}


_PREPARE = {"rows": _prepare_rows, "mesh": _prepare_mesh, "amr": _prepare_amr, "mm": _prepare_mm,
            "transfer": _prepare_transfer, "adjoint": _prepare_adjoint}
_RUN = {"rows": _run_rows, "mesh": _run_mesh, "amr": _run_amr, "mm": _run_mm, "transfer": _run_transfer,
        "adjoint": _run_adjoint}


def prepare(case, seed):
    return {"case": case, **_PREPARE[case["kind"]](case, seed)}


def run(state):
    return _RUN[state["case"]["kind"]](state["case"], state)


def work(case):
    """Every step reads the state and writes the next one (the global dt lies
    between two steps); the flops are counted from the scheme's formulas, each
    face once: about 90 for a first-order step with two HLLC faces per cell, 300
    for a second-order stage with slopes and reconstruction."""
    kind = case["kind"]
    if kind in ("rows", "mesh"):
        up = case["nx"] * case["ny"] * case["steps"]
        stages = 2 if case["accuracy"] == 2 and case["scheme"] == "heun" else 1
        per = 90 if case["accuracy"] == 1 else 300
        # five fields and the isolation counter in and out (MIXED: four FP64
        # conserved and five FP32 primitive fields)
        return {"bytes": up * (2 * 52 if kind == "mesh" else 2 * 44), "flops": up * stages * per}
    if kind == "amr":
        # the base mesh, and a band of some 24 finest cells along the interfaces
        rim = 2 * math.pi * sum(b[2] for b in BUBBLES)
        cells = case["n0"] ** 2 + 24 * rim * case["n0"] * 2 ** case["levels"]
        up = cells * case["adapts"] * 10
        return {"bytes": up * 2 * 44, "flops": up * 330}
    if kind == "mm":
        up = case["n"] ** 2 * case["steps"] * {"NONE": 1, "SIMPLE": 2, "STRANG": 3}[case["split"]]
        return {"bytes": up * 2 * 80, "flops": up * (150 if case["accuracy"] == 1 else 600)}
    if kind == "transfer":
        up = case["nx"] * case["ny"] * case["steps"] * (2 if case["split"] else 1)
        return {"bytes": up * 2 * 40, "flops": up * 20}
    up = case["nx"] * case["ny"] * case["steps"] * 2
    # each stage once forward and once reversed
    return {"bytes": up * 4 * 32, "flops": up * (300 + 700)}


# ---- the same by plain torch in 64 bits ---------------------------------------------------
def _limiter(name):
    zero = torch.zeros((), dtype=torch.float64, device=DEV)

    def phi(a, b):  # b * limiter(a, b)
        up = a * b > 0.0
        if name == "minmod":
            return torch.where(up, torch.where(a.abs() < b.abs(), a, b), zero)
        if name == "MC":
            m = torch.minimum(torch.minimum(2 * a.abs(), 2 * b.abs()), 0.5 * (a + b).abs())
            return torch.where(up, torch.sign(b) * m, zero)
        if name == "van Leer":
            return torch.where(up, 2 * a * b / torch.where(up, a + b, 1.0), zero)
        d = torch.where(up, a * a + b * b, 1.0)  # van Albada
        return torch.where(up, a * (a + b) / d * b, zero)
    return phi


class _Euler:
    """The single-material step on the unit square."""

    def __init__(self, case):
        self.c = case
        self.h = (1.0 / case["nx"], 1.0 / case["ny"])
        self.vol = self.h[0] * self.h[1]
        self.liquid = case.get("eos") == "stiffened"
        self.g, self.P0 = LIQUID if self.liquid else (GAMMA, 0.0)
        self.phi = _limiter(case["limiter"])

    def energy(self, r, p):
        return (p + self.g * self.P0) / ((self.g - 1.0) * r)

    def sound(self, r, p):
        return torch.sqrt(self.g * (p + self.P0) / r)

    def cons(self, w):
        r, u, v, p = w
        return torch.stack([r, r * u, r * v, r * (self.energy(r, p) + 0.5 * (u * u + v * v))])

    def prim(self, q):
        r, u, v = q[0], q[1] / q[0], q[2] / q[0]
        e = q[3] / r - 0.5 * (u * u + v * v)
        return torch.stack([r, u, v, (self.g - 1.0) * r * e - self.g * self.P0])

    def ghost(self, w, axis):
        """One layer of neighbours' values on each side of the axis."""
        d = axis + 1
        lo, hi = w.narrow(d, 0, 1).clone(), w.narrow(d, w.shape[d] - 1, 1).clone()
        if self.c["bounds"] == "periodic":
            lo, hi = hi, lo
        elif self.c["bounds"] == "wall":
            lo[1 + axis] *= -1.0
            hi[1 + axis] *= -1.0
        return torch.cat([lo, w, hi], d)

    def slopes(self, w, axis):
        """Half a cell's change of each value along the axis."""
        d, n = axis + 1, w.shape[axis + 1]
        z = self.ghost(w, axis)
        dl, dr = w - z.narrow(d, 0, n), z.narrow(d, 2, n) - w
        # the limited refit over both neighbours
        return 0.25 * (self.phi(dl, dr) + self.phi(dr, dl))

    def flux(self, w, axis):
        n, t = 1 + axis, 2 - axis
        r, un, p = w[0], w[n], w[3]
        f = [None] * 4
        f[0] = r * un
        f[n] = r * un * un + p
        f[t] = r * un * w[t]
        f[3] = (r * (self.energy(r, p) + 0.5 * (w[1] * w[1] + w[2] * w[2])) + p) * un
        return torch.stack(f)

    def riemann(self, L, R, axis):
        n, t = 1 + axis, 2 - axis
        cL, cR = self.sound(L[0], L[3]), self.sound(R[0], R[3])
        FL, FR, QL, QR = self.flux(L, axis), self.flux(R, axis), self.cons(L), self.cons(R)
        SL, SR = torch.minimum(L[n] - cL, R[n] - cR), torch.maximum(L[n] + cL, R[n] + cR)
        if self.c["flux"] == "HLL":
            SL, SR = torch.clamp(SL, max=0.0), torch.clamp(SR, min=0.0)
            return (SR * FL - SL * FR + SL * SR * (QR - QL)) / (SR - SL)
        aL, aR = L[0] * (SL - L[n]), R[0] * (SR - R[n])
        SC = (L[3] - R[3] + aR * R[n] - aL * L[n]) / (aR - aL)

        def star(W, S, a, Q):
            rs = a / (S - SC)
            f = [None] * 4
            f[0], f[n], f[t] = rs, rs * SC, rs * W[t]
            f[3] = rs * (Q[3] / W[0] + (SC - W[n]) * (SC + W[3] / a))
            return torch.stack(f)
        F = torch.where(SC >= 0.0, FL + SL * (star(L, SL, aL, QL) - QL), FR + SR * (star(R, SR, aR, QR) - QR))
        return torch.where(SL >= 0.0, FL, torch.where(SR <= 0.0, FR, F))

    def divergence(self, w, slopes):
        """Sum over the faces of area times flux out of every cell."""
        out = 0.0
        for axis in (0, 1):
            d, n = axis + 1, w.shape[axis + 1]
            if slopes is None:
                z = self.ghost(w, axis)
                lo, hi = z, z
            else:
                # states on the low and the high face of every cell; past a
                # boundary the mirror of the face's own state
                lo, hi = w - slopes[axis], w + slopes[axis]
                if self.c["bounds"] == "periodic":
                    lo, hi = self.ghost(lo, axis), self.ghost(hi, axis)
                else:
                    a, b = self.ghost(lo, axis), self.ghost(hi, axis)
                    m = a.shape[d]
                    lo = torch.cat([a.narrow(d, 0, m - 1), b.narrow(d, m - 1, 1)], d)
                    hi = torch.cat([a.narrow(d, 0, 1), b.narrow(d, 1, m - 1)], d)
            F = self.riemann(hi.narrow(d, 0, n + 1), lo.narrow(d, 1, n + 1), axis)
            out = out + (F.narrow(d, 1, n) - F.narrow(d, 0, n)) * self.h[1 - axis]
        return out

    def dt(self, w):
        return 0.4 * (min(self.h) / (torch.hypot(w[1], w[2]) + self.sound(w[0], w[3]))).min()

    def step(self, w):
        dt = self.dt(w)
        k = dt / self.vol
        q = self.cons(w)
        if self.c["accuracy"] == 1:
            return self.prim(q - k * self.divergence(w, None)), dt
        s = (self.slopes(w, 0), self.slopes(w, 1))
        if self.c["scheme"] == "heun":
            ws = self.prim(q - k * self.divergence(w, s))
            s = (self.slopes(ws, 0), self.slopes(ws, 1))
            return self.prim(0.5 * (q + self.cons(ws) - k * self.divergence(ws, s))), dt
        out = 0.0
        for axis in (0, 1):  # predictor: each cell's own face values
            out = out + (self.flux(w + s[axis], axis) - self.flux(w - s[axis], axis)) * self.h[1 - axis]
        wh = self.prim(q - 0.5 * k * out)
        return self.prim(q - k * self.divergence(wh, s)), dt


def _exact_euler(case, seed):
    f = _Euler(case)
    w = torch.stack([t.expand(case["nx"], case["ny"]) for t in _primitive(case, seed)])
    for _ in range(case["steps"]):
        w, dt = f.step(w)
    r, u, v, p = w
    five = torch.stack([r, u, v, p, f.energy(r, p)]).reshape(5, -1)
    return five, float(dt)


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    r, u, v, p = _primitive(case, seed)
    h = (1.0 / case["nx"], 1.0 / case["ny"])
    dt = 0.4 * min(h) / float((torch.hypot(u, v) + torch.sqrt(GAMMA * p / r)).max())
    r = r.clone().requires_grad_(True)
    g = torch.tensor(GAMMA, dtype=torch.float64, device=DEV, requires_grad=True)

    def prim(U, g):
        return U[0], U[1] / U[0], U[2] / U[0], (g - 1.0) * (U[3] - 0.5 * (U[1] * U[1] + U[2] * U[2]) / U[0])

    def half_slope(w, d):
        a, b = torch.roll(w, 1, d) - w, torch.roll(w, -1, d) - w
        return 0.25 * (a - b) * (2.0 * a * b - 1e-8) / (a * a + b * b + 1e-8)

    def flux(L, R, g):
        def side(w):
            rE = w[3] / (g - 1.0) + 0.5 * w[0] * (w[1] * w[1] + w[2] * w[2])
            Q = torch.stack([w[0], w[0] * w[1], w[0] * w[2], rE])
            F = torch.stack([Q[1], Q[1] * w[1] + w[3], Q[1] * w[2], (rE + w[3]) * w[1]])
            return Q, F, torch.sqrt(g * w[3] / w[0])
        (QL, FL, cL), (QR, FR, cR) = side(L), side(R)
        SL, SR = torch.minimum(L[1] - cL, R[1] - cR), torch.maximum(L[1] + cL, R[1] + cR)
        aL, aR = L[0] * (SL - L[1]), R[0] * (SR - R[1])
        SC = (L[3] - R[3] + aR * R[1] - aL * L[1]) / (aR - aL)

        def star(w, Q, S, a):
            rs = a / (S - SC)
            return torch.stack([rs, rs * SC, rs * w[2], rs * (Q[3] / w[0] + (SC - w[1]) * (SC + w[3] / a))])
        F = torch.where(SC >= 0.0, FL + SL * (star(L, QL, SL, aL) - QL), FR + SR * (star(R, QR, SR, aR) - QR))
        return torch.where(SL >= 0.0, FL, torch.where(SR <= 0.0, FR, F))

    def operator(U, g):
        w, out = prim(U, g), 0.0
        for d, (n, t) in enumerate(((1, 2), (2, 1))):
            s = [half_slope(x, d) for x in w]
            hi, lo = [x + y for x, y in zip(w, s)], [torch.roll(x - y, -1, d) for x, y in zip(w, s)]
            F = flux([hi[0], hi[n], hi[t], hi[3]], [lo[0], lo[n], lo[t], lo[3]], g)
            F = torch.stack([F[0], F[n], F[t], F[3]])
            out = out - (F - torch.roll(F, 1, d + 1)) / h[d]
        return out

    def step(U, g):
        Us = U + dt * operator(U, g)
        return 0.5 * (U + Us + dt * operator(Us, g))

    U = torch.stack([r, r * u, r * v, p / (g - 1.0) + 0.5 * r * (u * u + v * v)])
    for _ in range(case["steps"]):
        U = checkpoint(step, U, g, use_reentrant=False)
    cx, cy = _centres(case["nx"])[:, None], _centres(case["ny"])[None, :]
    probe = (cx >= 0.6) & (cx <= 0.7) & (cy >= 0.6) & (cy <= 0.7)
    J = (prim(U, g)[3] * probe).sum() / probe.sum()
    J.backward()
    return {"J": float(J), "drho": r.grad, "dgamma": float(g.grad)}


def exact(case, seed):
    """None for the kinds whose result has no short independent form: adaptive
    meshes, multi-material cells and VOF transport (their kernels restate
    whole mesh and geometry algorithms)."""
    if case["kind"] == "rows":
        five, dt = _exact_euler(case, seed)
        return {"state": five.reshape(-1), "wait": None, "dt": dt}
    if case["kind"] == "mesh":
        five, dt = _exact_euler(case, seed)
        return {"state": [x.cpu().numpy() for x in five], "dt": dt}
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    return None
