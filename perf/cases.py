"""Timed workloads of the hydro step, through the package's public entry points.

A case is a dict of plain values; `prepare` makes what a user's program holds
before the call, `run` is one pass of that program, `work` what the pass cannot
do without, and `exact` the same pass restated in plain torch (FP64, whole-array
operations in the formulas of the reference's subroutines).

The kinds stand for the ways the framework is used:

* `loop`      a driver that calls one step at a time and looks at the clock after
              each (the reference's main loop with its own work in between);
* `evolve`    a state resident on the device, advanced many steps between two
              looks at it (the bulk of every simulation);
* `restart`   a state handed over from the host, advanced, and looked at: the
              short runs of parameter studies, and the optional physics;
* `gravity`   a host-side potential solver coupled in before every step;
* `host`      a driver that keeps the state on the host between steps;
* `ensemble`  many boxes of several sizes advanced together;
* `gradient`  a differentiable run and its gradient.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from boxzyhydro_b200.adjoint import AdjointEngine, AdjointRun
from boxzyhydro_b200.batch import Batch
from boxzyhydro_b200.hydro import Hydro
from boxzyhydro_b200.params import HydroParams

# units%density (g/cm^3 per code density) and scale%rgas of the reference's code
# units, which the synthetic equation-of-state tables are written in
DENSITY_UNIT = 5.94327695e-07
RGAS = 8.254e7 / (1.496e13 / ((3600.0 * 365.25 * 24.0) / (2.0 * 3.1415926535897931))) ** 2

OPEN, CLOSED = "000000", "111111"


def listed():
    return [
        # the reference's shipped input file (an 8 x 200 x 1 Sod tube, walls all
        # round), driven step by step: the smallest call there is
        {"name": "loop_tube_4x196", "kind": "loop", "flow": "tube", "nx": 4, "ny": 196, "nz": 1,
         "walls": CLOSED, "h": 0.01, "cfl": 0.1, "gamma": 1.4, "steps": 16},
        # the 512-cell Sod tube of the tests and the benchmark, run in chunks
        {"name": "evolve_tube_512", "kind": "evolve", "flow": "tube", "nx": 512, "ny": 4, "nz": 4,
         "walls": CLOSED, "h": 1.0 / 512, "cfl": 0.1, "gamma": 1.4, "steps": 64},
        # a small open box of a parameter study: latency and launches count
        {"name": "restart_box_32", "kind": "restart", "flow": "turbulence", "nx": 32, "ny": 32,
         "nz": 32, "walls": OPEN, "h": 1.0 / 32, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 32},
        # odd sides, a cell size that is no power of two, walls on some sides
        {"name": "restart_ragged_75x61x47", "kind": "restart", "flow": "turbulence", "nx": 75,
         "ny": 61, "nz": 47, "walls": "011001", "h": 0.013, "cfl": 0.4, "gamma": 1.4, "steps": 32},
        # the benchmark's box: decaying turbulence, 256^3, resident on the device
        {"name": "evolve_box_256", "kind": "evolve", "flow": "turbulence", "nx": 256, "ny": 256,
         "nz": 256, "walls": OPEN, "h": 1.0 / 256, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 8},
        # the namelist's default walls in 3-D: a closed box
        {"name": "evolve_closed_96", "kind": "evolve", "flow": "turbulence", "nx": 96, "ny": 96,
         "nz": 96, "walls": CLOSED, "h": 1.0 / 96, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 16},
        # self-gravity: the host's potential goes in before every step
        {"name": "gravity_box_96", "kind": "gravity", "flow": "turbulence", "nx": 96, "ny": 96,
         "nz": 96, "walls": OPEN, "h": 1.0 / 96, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 8},
        # the tabulated equation of state (the namelist's default H2STAT is a table)
        {"name": "eos_box_96", "kind": "restart", "flow": "turbulence", "nx": 96, "ny": 96,
         "nz": 96, "walls": OPEN, "h": 1.0 / 96, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 16,
         "physics": "table"},
        # angular-momentum fluxing about an axis outside the box
        {"name": "angmom_box_96", "kind": "restart", "flow": "turbulence", "nx": 96, "ny": 96,
         "nz": 96, "walls": OPEN, "h": 1.0 / 96, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 16,
         "physics": "angmom"},
        # the host holds the state between steps: copies both ways in every call
        {"name": "host_box_128", "kind": "host", "flow": "turbulence", "nx": 128, "ny": 128,
         "nz": 128, "walls": OPEN, "h": 1.0 / 128, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 4},
        # the ensemble of Riemann problems, sides drawn per box, and the end states back
        {"name": "ensemble_12_boxes", "kind": "ensemble", "boxes": 12, "smallest": 32,
         "largest": 64, "steps": 100},
        # forward and backward of a checkpointed differentiable run
        {"name": "gradient_box_64", "kind": "gradient", "flow": "turbulence", "nx": 64, "ny": 64,
         "nz": 64, "walls": OPEN, "h": 1.0 / 64, "cfl": 0.4, "gamma": 5.0 / 3.0, "steps": 16,
         "snapshots": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "evolve", "evolve", "evolve", "restart", "restart", "gravity",
                       "host", "ensemble", "gradient"])
    if kind == "ensemble":
        smallest = rng.randint(16, 40)
        return {"kind": kind, "boxes": _log_int(rng, 4, 16), "smallest": smallest,
                "largest": smallest + rng.randint(8, 24), "steps": rng.randint(30, 100)}
    if kind in ("loop", "evolve") and rng.random() < 0.25:
        nx = _log_int(rng, 48, 1024)
        return {"kind": kind, "flow": "tube", "nx": nx, "ny": rng.randint(4, 12),
                "nz": rng.choice([1, 2, 4]), "walls": CLOSED, "h": 1.0 / nx, "cfl": 0.1,
                "gamma": rng.choice([1.4, 5.0 / 3.0]), "steps": rng.randint(8, 64)}
    most = {"loop": 64, "evolve": 224, "restart": 112, "gravity": 112, "host": 144,
            "gradient": 72}[kind]
    side = _log_int(rng, 20, most)
    n = [max(12, int(round(side * rng.uniform(0.75, 1.25)))) for _ in range(3)]
    walls = OPEN if rng.random() < 0.5 else "".join(rng.choice("01") for _ in range(6))
    if kind == "evolve" and rng.random() < 0.3:
        walls = CLOSED
    case = {"kind": kind, "flow": "turbulence", "nx": n[0], "ny": n[1], "nz": n[2],
            "walls": walls, "h": rng.choice([1.0 / 64, 1.0 / side, 0.01]), "cfl": 0.4,
            "gamma": rng.choice([1.4, 5.0 / 3.0]),
            "steps": max(1, min(rng.randint(4, 16), 130_000_000 // (n[0] * n[1] * n[2])))}
    if kind == "restart":
        case["steps"] = rng.randint(8, 32)
        physics = rng.choice(["", "", "table", "angmom"])
        if physics:
            # the angular-momentum pressure terms have a pole on the cell centre
            # that odd nx and ny put on the axis
            case.update(physics=physics, walls=OPEN, nx=n[0] + n[0] % 2)
    if kind == "gradient":
        case.update(walls=OPEN, steps=rng.randint(6, 16), snapshots=rng.randint(3, 8))
    if kind == "host":
        case["walls"] = OPEN
    return case


# ---------------------------------------------------------------- set-up

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _padded(case):
    """Cells per axis with ghosts: two per side, none in z below six planes."""
    nz = case["nz"] if case["nz"] < 6 else case["nz"] + 4
    return case["nx"] + 4, case["ny"] + 4, nz


def _params(case):
    nx, ny, nz = _padded(case)
    w = [c == "1" for c in case["walls"]]
    physics = case.get("physics", "")
    span = max(case["nx"], case["ny"], case["nz"]) * case["h"]
    return HydroParams(nx=nx, ny=ny, nz=nz, dx=case["h"], dy=case["h"], dz=case["h"],
                       cfl=case["cfl"], small_rho=1e-12, small_eps=1e-40, vlimit=10.0,
                       gammafix=case["gamma"], h2stat=1 if physics == "table" else -1,
                       fluxangmom=physics == "angmom", yoffset=0.75 * span,
                       no_outflow_xl=w[0], no_outflow_xr=w[1], no_outflow_yl=w[2],
                       no_outflow_yr=w[3], no_outflow_zl=w[4], no_outflow_zr=w[5],
                       endtime=1e30)


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _modes(gen, shape):
    """A random field's modes with power spectrum k^-2, and its wave vector."""
    dev = _device()
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device=dev, dtype=torch.float64))
    kz, ky = (torch.fft.fftfreq(n, 1.0 / n, device=dev, dtype=torch.float64) for n in shape[:2])
    kx = torch.fft.rfftfreq(shape[2], 1.0 / shape[2], device=dev, dtype=torch.float64)
    k = (kx[None, None, :], ky[None, :, None], kz[:, None, None])
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    k2[0, 0, 0] = 1.0
    f /= k2.sqrt()
    f[0, 0, 0] = 0.0
    return f, k, k2


def _smooth_noise(gen, shape):
    """A real random field with power spectrum k^-2, zero mean, unit variance."""
    x = torch.fft.irfftn(_modes(gen, shape)[0], s=shape)
    return x / x.std()


def _swirl(gen, shape):
    """A divergence-free random velocity, power spectrum k^-2, rms speed one."""
    f = []
    for _ in range(3):
        a, k, k2 = _modes(gen, shape)
        f.append(a)
    div = (k[0] * f[0] + k[1] * f[1] + k[2] * f[2]) / k2
    u = [torch.fft.irfftn(a - kk * div, s=shape) for a, kk in zip(f, k)]
    rms = torch.sqrt((u[0] ** 2 + u[1] ** 2 + u[2] ** 2).mean())
    return [a / rms for a in u]


def _interior(case, seed):
    """Conserved variables of the interior cells, (5, nz, ny, nx), made from the seed."""
    gen = _generator(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    if case["flow"] == "tube":
        # Sod's states on either side of the middle of the long axis, jittered by the seed
        jit = torch.rand(3, generator=gen, device=_device(), dtype=torch.float64).tolist()
        axis = 2 if case["nx"] >= case["ny"] else 1
        n = shape[axis]
        left = (torch.arange(n, device=_device()) < int(n * (0.4 + 0.2 * jit[0])))
        view = [1, 1, 1]
        view[axis] = n
        left = left.view(view).expand(shape)
        rho = torch.where(left, 1.0, 0.125 * (0.8 + 0.4 * jit[1])).to(torch.float64)
        p = torch.where(left, 1.0, 0.1 * (0.8 + 0.4 * jit[2])).to(torch.float64)
        u = [torch.zeros_like(rho) for _ in range(3)]
    else:
        # lognormal density, divergence-free velocities of rms Mach 1, smooth pressure
        rho = torch.exp(0.5 * _smooth_noise(gen, shape) - 0.125)
        p = torch.exp((0.2 if case["kind"] == "gradient" else 0.02) * _smooth_noise(gen, shape))
        u = [math.sqrt(case["gamma"]) * a for a in _swirl(gen, shape)]
    e = p / (case["gamma"] - 1.0) + rho * 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    return torch.stack([rho, rho * u[0], rho * u[1], rho * u[2], e])


def _with_ghosts(case, q):
    """Ghost layers: a copy of the last cell, or its mirror image at a wall."""
    for axis, n, lo, hi, flip in ((3, case["nx"], 0, 1, 1), (2, case["ny"], 2, 3, 2),
                                  (1, case["nz"], 4, 5, 3)):
        if axis == 1 and case["nz"] < 6:
            continue
        wl, wh = case["walls"][lo] == "1", case["walls"][hi] == "1"
        idx = ([1, 0] if wl else [0, 0]) + list(range(n)) + \
              ([n - 1, n - 2] if wh else [n - 1, n - 1])
        q = q.index_select(axis, torch.tensor(idx, device=q.device))
        sign = torch.ones(n + 4, device=q.device, dtype=q.dtype)
        sign[:2] = -1.0 if wl else 1.0
        sign[n + 2:] = -1.0 if wh else 1.0
        view = [1] * 3
        view[axis - 1] = n + 4
        q = torch.cat([q[:flip], (q[flip] * sign.view(view))[None], q[flip + 1:]])
    return q


def _host_arrays(case, q, pinned=False):
    """cons (ng,5), u (ng,3) and p (ng,) in the reference's layout, on the host."""
    q = q.reshape(5, -1)
    u = q[1:4] / q[0]
    p = (case["gamma"] - 1.0) * (q[4] - q[0] * 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))
    out = []
    for a in (q.t().contiguous(), u.t().contiguous(), p):
        b = torch.empty(a.shape, dtype=torch.float64, pin_memory=pinned)
        out.append(b.copy_(a))
    return out


def _table():
    """Equation-of-state tables in the layout of the reference's eos module:
    log-spaced energies per density row, smooth gamma and mean molecular weight."""
    neos, nrho, low, step = 40, 9, -9.0, 0.5
    j = np.arange(1, nrho + 1)
    i = np.arange(1, neos + 1)[:, None]
    deng = 0.05 + 0.002 * j
    eng = (0.1 * (1.0 + 0.1 * j))[None, :] * 10.0 ** ((i - 1) * deng[None, :])
    gam = 1.5 + 0.1 * np.sin(0.2 * i + j[None, :])
    muc = 2.3 - 0.5 * i / neos + 0.01 * j[None, :]
    return dict(neos=neos, neos_rho=nrho, log_rho_eos_low=low, drho_eos=step,
                density_unit=DENSITY_UNIT, tk_bgrnd=1e-6, eng_table2=eng, gamma_table2=gam,
                muc_table2=muc, tk_table2=(gam - 1.0) * eng * muc / RGAS,
                rho_table=10.0 ** (low + (j - 1) * step) / DENSITY_UNIT, deng_eos_array=deng)


def _centres(case, axis, ghosts=0):
    """Cell-centre coordinates along an axis (0 = x), the box's middle at zero."""
    n = (case["nx"], case["ny"], case["nz"])[axis] + 2 * ghosts
    i = torch.arange(n, device=_device(), dtype=torch.float64)
    return case["h"] * (i - (n - 1) / 2.0)


def _potential(case, seed, step):
    """A softened point mass wandering about the box's middle, all cells, (nz, ny, nx)."""
    gen = _generator(seed + 77)
    s = torch.rand(3, generator=gen, device=_device(), dtype=torch.float64).tolist()
    g = 0 if case["nz"] < 6 else 2
    x, y, z = (_centres(case, 0, 2), _centres(case, 1, 2), _centres(case, 2, g))
    span = case["nx"] * case["h"]
    c = [span * (0.1 * (v - 0.5) + 0.01 * step) for v in s]
    r2 = ((x - c[0]) ** 2)[None, None, :] + ((y - c[1]) ** 2)[None, :, None] + \
         ((z - c[2]) ** 2)[:, None, None]
    return -0.05 / torch.sqrt(r2 / span ** 2 + 0.02)


def _boxes(case, seed):
    """The ensemble's boxes: one Riemann problem each, along a drawn axis."""
    rng = np.random.default_rng(int(seed) * 7919 + case["boxes"])
    sizes = np.random.default_rng(case["boxes"])
    out = []
    for _ in range(case["boxes"]):
        n = int(sizes.integers(case["smallest"], case["largest"] + 1))
        lr = [(float(np.exp(rng.uniform(-1, 1))), float(rng.uniform(-0.5, 0.5)),
               float(np.exp(rng.uniform(-1, 1)))) for _ in range(2)]
        out.append((dict(kind="ensemble", nx=n, ny=n, nz=n, walls=OPEN, h=1.0 / n, cfl=0.1,
                         gamma=float(rng.choice([1.4, 5.0 / 3.0]))), int(rng.integers(0, 3)), lr))
    return out


def _riemann(box, axis, lr):
    n = box["nx"]
    q = torch.zeros(5, n, n, n, dtype=torch.float64, device=_device())
    view = [1, 1, 1]
    view[2 - axis] = n
    side = (torch.arange(n, device=_device()) >= n // 2).long().view(view).expand(n, n, n)
    rho, v, p = (torch.tensor([lr[0][k], lr[1][k]], dtype=torch.float64, device=_device())[side]
                 for k in range(3))
    q[0] = rho
    q[1 + axis] = rho * v
    q[4] = p / (box["gamma"] - 1.0) + 0.5 * rho * v * v
    return q


def _end_gradient(case, seed):
    """The gradient of a loss in the end state, all cells, as the run's planes."""
    nx, ny, nz = _padded(case)
    return torch.randn((5, nx * ny * nz), generator=_generator(seed + 55), device=_device(),
                       dtype=torch.float64)


class _Planes:
    """A view of a handle's planes; tensors made from it keep the handle alive."""

    def __init__(self, hydro):
        self.hydro = hydro
        ptr, ngrid = hydro.device_cons()
        self.__cuda_array_interface__ = {"shape": (5, ngrid), "typestr": "<f8", "version": 2,
                                         "data": (ptr, False)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        boxes = _boxes(case, seed)
        batch = Batch([_params(b) for b, _, _ in boxes])
        cons = []
        for k, (b, axis, lr) in enumerate(boxes):
            c = _host_arrays(b, _with_ghosts(b, _riemann(b, axis, lr)))[0]
            batch.upload(k, c.numpy())
            cons.append(c.numpy())
        return {"case": case, "batch": batch, "cons": cons}
    q = _with_ghosts(case, _interior(case, seed))
    if kind == "gradient":
        engine = AdjointEngine(_params(case), case["steps"], case["snapshots"])
        return {"case": case, "engine": engine, "cons": q.reshape(5, -1).contiguous(),
                "g": _end_gradient(case, seed)}
    state = {"case": case, "hydro": Hydro(_params(case))}
    if case.get("physics") == "table":
        state["hydro"].set_eos_table(_table())
    state["cons"], state["u"], state["p"] = _host_arrays(case, q, pinned=kind in ("restart", "host"))
    if kind == "gravity":
        state["phi"] = [_potential(case, seed, k).cpu().pin_memory().numpy().reshape(-1)
                        for k in range(case["steps"])]
    if kind == "host":
        state["hydro"].upload_conserved(state["cons"].numpy())
    elif kind != "restart":
        state["hydro"].upload(state["cons"].numpy(), state["u"].numpy(), state["p"].numpy())
    return state


def _look(hydro):
    """The conserved planes where they are, on the device."""
    return torch.as_tensor(_Planes(hydro), device="cuda")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        b = state["batch"]
        b.run(case["steps"])
        return [[b.download(k)[0], b.clock(k)["time"]] for k in range(b.nbox)]
    if kind == "gradient":
        c0 = state["cons"].detach().requires_grad_(True)
        out = AdjointRun.apply(c0, state["engine"])
        out.backward(state["g"])
        return {"out": out.detach(), "grad": c0.grad}
    h = state["hydro"]
    if kind == "loop":
        times = []
        for _ in range(case["steps"]):
            h.step()
            times.append(h.clock()["time"])
        return {"cons": _look(h), "times": times}
    if kind == "evolve":
        h.run(nsteps=case["steps"])
        return {"cons": _look(h), "time": h.clock()["time"]}
    if kind == "restart":
        h.upload(state["cons"].numpy(), state["u"].numpy(), state["p"].numpy())
        h.set_clock(0.0, 0.0, 0)
        h.run(nsteps=case["steps"])
        return {"cons": _look(h), "time": h.clock()["time"]}
    if kind == "gravity":
        for k in range(case["steps"]):
            h.set_phi(state["phi"][k])
            h.step()
        return {"cons": _look(h), "time": h.clock()["time"]}
    for _ in range(case["steps"]):  # host
        h.step_host(state["cons"].numpy())
    return {"cons": state["cons"], "time": h.clock()["time"]}


def work(case):
    if case["kind"] == "ensemble":
        cells = sum(b["nx"] ** 3 for b, _, _ in _boxes(case, 0))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    # per cell and step: five doubles read and written; about 950 operations
    # (three reconstructions, three faces and the update, twice), a division or
    # square root counted as one; the gradient's backward counts as twice a step
    passes = 3 if case["kind"] == "gradient" else 1
    return {"bytes": 80.0 * cells * case["steps"] * passes,
            "flops": 950.0 * cells * case["steps"] * passes}


# ---------------------------------------------------------------- the step in plain torch

THETA = 1.25
FLOOR_RHO, FLOOR_EPS = 1e-12, 1e-40


def _thermal(q, u):
    """Internal energy per volume, above its floor."""
    return (q[4] - 0.5 * q[0] * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)).clamp(min=FLOOR_EPS)


def _slope(a, b, c):
    d1, d2, d3 = THETA * (b - a), 0.5 * (c - a), THETA * (c - b)
    m = torch.where(d1.abs() < d2.abs(), d1, d2)
    m = torch.where(m.abs() < d3.abs(), m, d3)
    return torch.where((b - a) * (c - b) > 0, m, torch.zeros_like(m))


class _Exact:
    """The fixed-dt step on interior arrays (nz, ny, nx)."""

    def __init__(self, case):
        self.case = case
        self.h = case["h"]
        self.gam = case["gamma"]
        self.threed = case["nz"] >= 6
        self.physics = case.get("physics", "")
        self.walls = [c == "1" for c in case["walls"]]
        if self.physics == "table":
            t = _table()
            self.tab = {k: torch.as_tensor(v, device=_device()) if isinstance(v, np.ndarray) else v
                        for k, v in t.items()}
        if self.physics == "angmom":
            self.yoff = _params(case).yoffset

    def eos(self, rho, eps):
        """Pressure and gamma of state(): fixed gamma, or the tables' bilinear look-up."""
        if self.physics != "table":
            return eps * (self.gam - 1.0), None
        t = self.tab
        nr, ne = t["neos_rho"], t["neos"]
        ir = ((torch.log10(rho * t["density_unit"]) - t["log_rho_eos_low"]) / t["drho_eos"]).trunc()
        ir = ir.long().clamp(0, nr - 1)
        jr = (ir + 1).clamp(max=nr - 1)
        eng = eps / rho
        e1 = t["eng_table2"][0]
        ie = ((torch.log10(eng) - torch.log10(e1[ir])) / t["deng_eos_array"][ir]).trunc().long()
        eng = torch.where(ie > ne - 2, t["eng_table2"][ne - 1][ir], eng)
        eng = torch.where((ie < 0) | (eng < e1[ir]), e1[ir], eng)
        ie = ie.clamp(0, ne - 2)

        def row(name, r):
            e = t["eng_table2"]
            f = t[name]
            return f[ie, r] + (f[ie + 1, r] - f[ie, r]) / (e[ie + 1, r] - e[ie, r]) * (eng - e[ie, r])

        def both(name):
            a = row(name, ir)
            dr = t["rho_table"][jr] - t["rho_table"][ir]
            w = torch.where(dr == 0, torch.zeros_like(rho), (rho - t["rho_table"][ir]) /
                            torch.where(dr == 0, torch.ones_like(dr), dr))
            return a + (row(name, jr) - a) * w

        gam, mu, tk = both("gamma_table2"), both("muc_table2"), both("tk_table2")
        return rho * tk * RGAS / mu, gam

    def rate(self, q):
        u = [q[k] / q[0] for k in (1, 2, 3)]
        p, gam = self.eos(q[0], _thermal(q, u))
        c = torch.sqrt((self.gam if gam is None else gam) * p / q[0])
        return ((3.0 * c + u[0].abs() + u[1].abs() + u[2].abs()) / self.h).max()

    def ghosted(self, fields, axis):
        """Two ghost cells on either side of one axis (0 = x): copies, or mirror
        images with the normal velocity reversed."""
        dim = 2 - axis
        n = fields["d"].shape[dim]
        wl, wh = self.walls[2 * axis], self.walls[2 * axis + 1]
        idx = ([1, 0] if wl else [0, 0]) + list(range(n)) + \
              ([n - 1, n - 2] if wh else [n - 1, n - 1])
        idx = torch.tensor(idx, device=fields["d"].device)
        sign = torch.ones(n + 4, device=idx.device, dtype=torch.float64)
        sign[:2] = -1.0 if wl else 1.0
        sign[n + 2:] = -1.0 if wh else 1.0
        view = [1, 1, 1]
        view[dim] = n + 4
        out = {k: v.index_select(dim, idx) for k, v in fields.items()}
        out["u%d" % axis] = out["u%d" % axis] * sign.view(view)
        return out

    def polar(self, m1, m2, axis=None):
        """Radial and angular momenta about the axis through (0, -yoffset)."""
        gx, gy = 2 if axis == 0 else 0, 2 if axis == 1 else 0
        x = _centres(self.case, 0, gx)[None, None, :]
        y = _centres(self.case, 1, gy)[None, :, None] + self.yoff
        r = torch.sqrt(x * x + y * y)
        return (m1 * x + m2 * y) / r, x * m2 - y * m1, x, y, r

    def divergence(self, q, u, p, gam, dt):
        """Sum over the axes of the flux differences of (rho, m, E), over h."""
        d = q[0]
        eps = _thermal(q, u)
        c = torch.sqrt((self.gam if gam is None else gam) * p / d)
        cell = {"d": d, "u0": u[0], "u1": u[1], "u2": u[2], "p": p, "e": eps, "c": c}
        if gam is not None:
            cell["g"] = gam
        total = [torch.zeros_like(d) for _ in range(5)]
        for axis in range(3 if self.threed else 2):
            dim = 2 - axis
            n = d.shape[dim]
            w = self.ghosted(cell, axis)
            if self.physics == "angmom":
                w["r"], w["a"] = self.polar(w["d"] * w["u0"], w["d"] * w["u1"], axis)[:2]
            at = lambda f, k, m: f.narrow(dim, k, m)
            ud, c1 = at(w["u%d" % axis], 1, n + 2), at(w["c"], 1, n + 2)
            hp = 0.5 * (1.0 - (ud + c1).clamp(min=0.0) * dt / self.h)
            hm = 0.5 * (-1.0 - (ud - c1).clamp(max=0.0) * dt / self.h)
            inner = torch.ones(n + 2, device=d.device, dtype=torch.float64)
            inner[0] = inner[-1] = 0.0  # a ghost cell has no slope
            view = [1, 1, 1]
            view[dim] = n + 2
            inner = inner.view(view)
            left, right = {}, {}
            for k, f in w.items():
                if k == "c":
                    continue
                s = _slope(at(f, 0, n + 2), at(f, 1, n + 2), at(f, 2, n + 2)) * inner
                mid = at(f, 1, n + 2)
                left[k] = at(mid + hp * s, 0, n + 1)
                right[k] = at(mid + hm * s, 1, n + 1)
            sides = []
            for f in (left, right):
                v = f["u%d" % axis]
                a = torch.sqrt((f["g"] if "g" in f else self.gam) * f["p"] / f["d"])
                e = f["e"] + 0.5 * f["d"] * (f["u0"] ** 2 + f["u1"] ** 2 + f["u2"] ** 2)
                sides.append((f, v, a, e))
            (fl, vl, al, el), (fr, vr, ar, er) = sides
            ap = torch.maximum((vr + ar).clamp(min=0.0), vl + al)
            am = torch.maximum((-(vr - ar)).clamp(min=0.0), -(vl - al))

            def hll(sl, sr, gl, gr):
                return (ap * gl + am * gr - ap * am * (sr - sl)) / (ap + am)

            pairs = [(fl["d"], fr["d"], 0.0, 0.0)]
            for k in range(3):
                own = 1.0 if k == axis else 0.0
                pairs.append((fl["d"] * fl["u%d" % k], fr["d"] * fr["u%d" % k],
                              own * fl["p"], own * fr["p"]))
            flux = [hll(sl, sr, sl * vl + xl, sr * vr + xr) for sl, sr, xl, xr in pairs]
            flux.append(hll(el, er, (el + fl["p"]) * vl, (er + fr["p"]) * vr))
            for k in range(5):
                lo, hi = at(flux[k], 0, n), at(flux[k], 1, n)
                if self.physics == "angmom" and k in (1, 2):
                    # the pressure terms are taken at the centre of the updated cell
                    x = _centres(self.case, 0)[None, None, :]
                    y = _centres(self.case, 1)[None, :, None]
                    r = torch.sqrt(x * x + y * y)
                    if axis == 2:
                        t = 0.0
                    elif k == 1:
                        t = (x if axis == 0 else y) / r
                    else:
                        t = -y if axis == 0 else x
                    name = "r" if k == 1 else "a"

                    def face(first):
                        ql, qr, pl, pr, v1, v2, bp, bm = (at(z, first, n) for z in (
                            fl[name], fr[name], fl["p"], fr["p"], vl, vr, ap, am))
                        return (bp * (pl * t + ql * v1) + bm * (pr * t + qr * v2) -
                                bp * bm * (qr - ql)) / (bp + bm)

                    lo, hi = face(0), face(1)
                total[k] = total[k] + (hi - lo) / self.h
        return total

    def kick(self, q, g, v, dt):
        """source(): momenta, and the work done with velocity v, above the energy's floor."""
        if g is None:
            g = (0.0, 0.0, 0.0)
        m = [q[1 + k] + q[0] * g[k] * dt for k in range(3)]
        k = 0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / q[0]
        e = q[4] - k + dt * q[0] * (v[0] * g[0] + v[1] * g[1] + v[2] * g[2])
        return [q[0], *m, e.clamp(min=FLOOR_EPS) + k]

    def step(self, q, dt, force=None):
        vel = lambda a: [a[k] / a[0] for k in (1, 2, 3)]
        old = vel(q)
        q0 = self.kick(q, force, old, 0.5 * dt)
        u0 = vel(q0)
        p, gam = self.eos(q0[0], _thermal(q0, old))
        div = self.divergence(q0, u0, p, gam, dt)
        q1 = self.update(q0, q0, div, dt, 1.0)
        # state() of the second stage still reads the velocities of the first
        p, gam = self.eos(q1[0], _thermal(q1, u0))
        div = self.divergence(q1, vel(q1), p, gam, dt)
        q2 = self.update(q0, q1, div, dt, 0.5)
        return self.kick(q2, force, vel(q2), 0.5 * dt)

    def update(self, q0, q1, div, dt, half):
        a, b = list(q0), list(q1)
        if self.physics == "angmom":
            a[1], a[2], x, y, r = self.polar(q0[1], q0[2])
            b[1], b[2] = self.polar(q1[1], q1[2])[:2]
        n = [(s - dt * f) if half == 1.0 else 0.5 * (s + t - dt * f) for s, t, f in zip(a, b, div)]
        if self.physics == "angmom":
            n[1], n[2] = (n[1] * x - n[2] * y / r) / r, (n[1] * y + n[2] * x / r) / r
        n[0] = n[0].clamp(min=FLOOR_RHO)
        k = 0.5 * (n[1] ** 2 + n[2] ** 2 + n[3] ** 2) / n[0]
        n[4] = torch.where(n[4] < 0, k + FLOOR_EPS, n[4])
        return n

    def run(self, q, steps, phis=None, dts=None):
        """`steps` steps from rest of the clock; the times after each, and the dts."""
        q, t, last, times, used = list(q), 0.0, 0.0, [], []
        for k in range(steps):
            if dts is None:
                dt = float(self.case["cfl"] / self.rate(q))
                dt = min(dt, 1.1 * last) if k and last > 0 else dt
            else:
                dt = dts[k]
            last = dt
            force = None
            if phis is not None:
                f = phis[k]
                m = (slice(2, -2),) * 3
                force = [-(f.roll(-1, 2 - a) - f.roll(1, 2 - a))[m] / (2.0 * self.h)
                         for a in range(3)]
            q = self.step(q, dt, force)
            t += dt
            times.append(t)
            used.append(dt)
        return torch.stack(q), times, used


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for b, axis, lr in _boxes(case, seed):
            q, times, _ = _Exact(b).run(_riemann(b, axis, lr), case["steps"])
            out.append([_with_ghosts(b, q).reshape(5, -1).t().contiguous().cpu(), times[-1]])
        return out
    e = _Exact(case)
    q0 = _interior(case, seed)
    if kind == "gradient":
        with torch.no_grad():
            _, _, dts = e.run(q0, case["steps"])
            states = [list(q0)]
            for dt in dts:
                states.append(e.step(states[-1], dt))
        nx, ny, nz = _padded(case)
        lam = _end_gradient(case, seed).reshape(5, nz, ny, nx)[_core(case)].contiguous()
        for dt, q in zip(reversed(dts), reversed(states[:-1])):
            q = torch.stack(q).requires_grad_(True)
            torch.stack(e.step(list(q), dt)).backward(lam)
            lam = q.grad
        grad = torch.zeros((5, nz, ny, nx), device=lam.device, dtype=lam.dtype)
        grad[_core(case)] = lam
        return {"out": _with_ghosts(case, torch.stack(states[-1])).reshape(5, -1),
                "grad": grad.reshape(5, -1)}
    phis = None
    if kind == "gravity":
        phis = [_potential(case, seed, k) for k in range(case["steps"])]
    q, times, _ = e.run(q0, case["steps"], phis)
    cons = _with_ghosts(case, q).reshape(5, -1)
    if kind == "loop":
        return {"cons": cons, "times": times}
    if kind == "host":
        return {"cons": cons.t().contiguous().cpu(), "time": times[-1]}
    return {"cons": cons, "time": times[-1]}


def _core(case):
    z = slice(None) if case["nz"] < 6 else slice(2, -2)
    return (slice(None), z, slice(2, -2), slice(2, -2))
