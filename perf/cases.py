"""The work that a program using this framework has it do, as timed and checked cases.

Every case is one whole call a user makes through the Python package (tinymd.Simulation over the
md_* C ABI, tinymd.adjoint): host arrays in, the grid set up, lists built, K timesteps, host arrays
out.  The library owns one grid per process, as the md driver does, so a pass over new inputs makes
the grid anew; only the differentiable form keeps its grid between calls, as a training loop does.

kind "run"      Simulation(...), run(dt, steps), arrays(), close()
     "monitor"  the same with the energy / virial / kinetic sums read every 10 steps (md --thermo)
     "evaluate" the forces of a given configuration: Simulation(...), arrays(), close()
     "adjoint"  TrajectoryLoss forward and backward on a kept grid

The FP64 form ("f64") hands out FP64 arrays.  The mixed form's pair forces are FP32, so its frame is
handed on in FP32, as trajectory frames are stored.  Positions and velocities are the whole state of
a run; forces are returned where the run is FP64 and by the evaluations (a pair that crosses the
truncated cutoff jumps by 0.039, so the mixed form's last forces after many steps of a chaotic
system say nothing about the arithmetic).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "molecular-dynamics_b200"))

import tinymd  # noqa: E402
from tinymd import adjoint  # noqa: E402

LATTICE = 1.6796                   # the md driver's lattice constant (reduced density 0.8442)
SKIN = 0.3
REBUILD = 20                       # steps between list builds (driver default)
READ_EVERY = 10                    # steps between reads of the sums ("monitor")
LJ = {"cutoff": 2.5, "dt": 0.005}  # eps = sigma = 1
DEM = {"cutoff": 1.2, "dt": 0.001, "params": (0.1, 0.1, 100.0, 0.5), "radius": 0.6}


def case(name, kind, setup, cells, steps, form="f64", half=False):
    c = {"kind": kind, "setup": setup, "nx": cells[0], "ny": cells[1], "nz": cells[2], "steps": steps, "form": form,
         "half": half}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest periodic box: a long run of a test system, one launch per step
        case("lj_f64_256", "run", "default", (4, 4, 4), 1000),
        # the small regression system of the tests, mixed form
        case("lj_mixed_2k", "run", "default", (8, 8, 8), 100, "mixed"),
        # single-point forces of an odd-sized configuration (scoring, fitting)
        case("evaluate_mixed_5k", "evaluate", "default", (13, 11, 9), 0, "mixed"),
        # a system of the differentiable form's size, the driver's default 100 steps
        case("lj_mixed_16k", "run", "default", (16, 16, 16), 100, "mixed"),
        # a ragged box watched by its energies: the driver's --thermo 10
        case("monitor_f64_30k", "monitor", "default", (23, 19, 17), 200),
        # the headline system (32^3 cells, full lists), FP64 form
        case("lj_f64_131k", "run", "default", (32, 32, 32), 500),
        # the same in the mixed form, the driver's default 100 steps
        case("lj_mixed_131k", "run", "default", (32, 32, 32), 100, "mixed"),
        # half lists that keep the pairs across the periodic boundary
        case("lj_half_f64_131k", "run", "default", (32, 32, 32), 100, half=True),
        # the half-filled box at 64^3: lists larger than L2, empty cells beside full ones
        case("lj_mixed_524k", "run", "half", (64, 64, 64), 100, "mixed"),
        # granular gas under the contact model, FP64
        case("dem_f64_261k", "run", "granular_gas", (48, 48, 48), 300),
        # the diagonally split FCC bed, mixed form
        case("dem_mixed_223k", "run", "granular_gas_fcc", (48, 48, 48), 100, "mixed"),
        # one training step of the differentiable form: loss, then all gradients
        case("adjoint_16k", "adjoint", "default", (16, 16, 16), 100),
    ]


def _atoms(c):
    sites = c["nx"] * c["ny"] * c["nz"]
    return {"default": 4.0, "half": 2.0, "granular_gas": LATTICE ** 3 / 2, "granular_gas_fcc": 2.0}[c["setup"]] * sites


def draw(rng):
    kind, setup, form, half = rng.choice([
        ("run", "default", "f64", False), ("run", "default", "mixed", False), ("run", "default", "mixed", False),
        ("run", "half", "f64", False), ("run", "half", "mixed", False), ("run", "default", "f64", True),
        ("run", "granular_gas", "f64", False), ("run", "granular_gas_fcc", "mixed", False),
        ("run", "granular_gas", "mixed", False), ("run", "granular_gas_fcc", "f64", False),
        ("monitor", "default", "f64", False), ("evaluate", "default", "mixed", False),
        ("evaluate", "default", "f64", False), ("adjoint", "default", "f64", False)])
    small = {"half": 8, "granular_gas": 6, "granular_gas_fcc": 6}.get(setup, 4)
    side = math.exp(rng.uniform(math.log(small), math.log(16 if kind == "adjoint" else 40)))
    cells = [max(small, min(64, int(round(side * rng.uniform(0.75, 1.3))))) for _ in range(3)]
    if kind == "adjoint":
        while cells[0] * cells[1] * cells[2] > 4096:
            cells[cells.index(max(cells))] -= 1
    # FP64 full-list runs go on for as long as a listed one; the others keep the driver's 100 steps
    long = kind == "run" and form == "f64" and not half
    steps = {"evaluate": 0, "monitor": 10 * rng.randint(6, 20), "adjoint": rng.randint(30, 100)}.get(
        kind, rng.randint(100, 400) if long else rng.randint(50, 100))
    c = case(None, kind, setup, cells, steps, form, half)
    return dict(c, steps=min(steps, int(6.5e7 / _atoms(c)))) if steps else c


# ---- inputs -------------------------------------------------------------------------------------
def _model(c):
    return DEM if c["setup"].startswith("granular") else LJ


def _inputs(c, seed):
    """(masses, positions, velocities, world, rank) as host arrays: the setup's sites displaced a
    little, a Maxwell distribution of velocities (T = 1.44 for LJ, slow grains for DEM)."""
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    m, x, v, world, rank = tinymd.setup_particles(c["setup"], (c["nx"], c["ny"], c["nz"]), LATTICE)
    lo, length = world[0::2], world[1::2] - world[0::2]
    dem = _model(c) is DEM
    x = lo + np.mod(x + rng.normal(0.0, 0.005 if dem else 0.02, x.shape) - lo, length)
    v = rng.normal(0.0, 1.0, x.shape)
    v -= v.mean(axis=0)
    v *= math.sqrt((0.01 if dem else 1.44) * (3 * len(m) - 3) / np.sum(v * v))
    return m, x, v, world, rank


_grid = None  # what the process's one grid was made for, where a program keeps it (adjoint)


def _open(c, inputs, precision):
    global _grid
    _grid = None
    lib = tinymd.load()
    model = _model(c)
    lib.md_set_precision(precision)
    lib.md_set_half_mode(1 if c["half"] else 0)
    lib.md_set_thermo(1 if c["kind"] == "monitor" else 0)
    more = {}
    if model is DEM:
        lib.md_set_dem_model(1, DEM["radius"])
        more = {"force_field": "dem", "dem": DEM["params"]}
    else:
        lib.md_set_dem_model(0, 1.0)
    return tinymd.Simulation(lib, *inputs, cutoff=model["cutoff"], skin=SKIN, half=c["half"], reneigh=REBUILD, **more)


def _adjoint_grid(c, place):
    """The kept grid of the differentiable form (lattice positions; velocities are an input)."""
    global _grid
    key = (c["nx"], c["ny"], c["nz"])
    if _grid != key:
        _open(c, place, 0)
        _grid = key


def prepare(c, seed):
    state = {"case": c, "lib": tinymd.load()}
    if c["kind"] != "adjoint":
        return dict(state, inputs=_inputs(c, seed))
    m, _, v, world, rank = _inputs(c, seed)
    place = tinymd.setup_particles("default", (c["nx"], c["ny"], c["nz"]), LATTICE)
    _adjoint_grid(c, place)
    eps, sigma = _parameters(seed)
    return dict(state, place=place, v0=torch.from_numpy(v).requires_grad_(),
                eps=torch.tensor(eps, dtype=torch.float64, requires_grad=True),
                sigma=torch.tensor(sigma, dtype=torch.float64, requires_grad=True))


def _parameters(seed):
    r = np.random.default_rng(seed + 1)
    return float(r.uniform(0.97, 1.03)), float(r.uniform(0.995, 1.005))


# ---- one pass -----------------------------------------------------------------------------------
def run(state):
    c, lib = state["case"], state["lib"]
    if c["kind"] == "adjoint":
        _adjoint_grid(c, state["place"])
        adjoint.configure(lib, steps=c["steps"], reneigh=REBUILD, dt=LJ["dt"], cutoff=LJ["cutoff"], skin=SKIN,
                          precision=0, shifted_energy=True)
        loss = adjoint.TrajectoryLoss.apply(state["v0"], state["eps"], state["sigma"], lib)
        return [loss.detach(), *torch.autograd.grad(loss, [state["v0"], state["eps"], state["sigma"]])]
    mixed = c["form"] == "mixed"
    sim = _open(c, state["inputs"], 1 if mixed else 0)
    dt = _model(c)["dt"]
    sums = []
    if c["kind"] == "monitor":
        ticket = None
        for _ in range(c["steps"] // READ_EVERY):
            sim.run(dt, READ_EVERY)
            if ticket is not None:
                sums.append(_fetch(lib, ticket))
            ticket = lib.md_thermo_request()
        sums.append(_fetch(lib, ticket))
    elif c["steps"]:
        sim.run(dt, c["steps"])
    _, x, v, f = sim.arrays()
    sim.close()
    if c["kind"] == "evaluate":
        return [torch.from_numpy(f).float() if mixed else f]
    if mixed:
        return [torch.from_numpy(x).float(), torch.from_numpy(v).float()]
    return [x, v, f] + ([np.stack(sums)] if sums else [])


def _fetch(lib, ticket):
    out = np.zeros(4)
    lib.md_thermo_fetch(ticket, tinymd.ptr(out))
    return out


def work(c):
    """State in and out once, and per step the state read and written once and each pair evaluated
    once per atom (list pairs: distance and test; pairs inside the cutoff: force and sum)."""
    n, model = _atoms(c), _model(c)
    rho = 0.65 if c["setup"] == "granular_gas" else 0.8442
    ball = 4.0 / 3.0 * math.pi * rho
    near, inside = ball * (model["cutoff"] + SKIN) ** 3, ball * model["cutoff"] ** 3
    if model is DEM:  # ordered beds: the first shell
        near = inside = 6 if c["setup"] == "granular_gas" else 12
    pair = near * 8 + inside * (15 if model is LJ else 45)
    if c["half"]:
        pair /= 2
    wide = 4 if c["form"] == "mixed" else 8
    out = 3 * wide * (1 if c["kind"] == "evaluate" else 2 if c["form"] == "mixed" else 3)
    evals = c["steps"] + 1
    total = {"bytes": n * (56 + out + 96.0 * c["steps"]), "flops": n * pair * evals}
    if c["kind"] == "adjoint":  # forward, recomputation, and one product with the force's derivative per step
        total = {"bytes": n * (48 + 96.0 * 3 * c["steps"]), "flops": n * (2 * pair + near * 8 + inside * 50) * evals}
    return total


# ---- the same in 64 bits, in plain torch --------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pairs(x, lo, length, reach):
    """All ordered pairs (i, j) whose nearest images are within `reach`, and the image shift of j in
    box lengths per axis, by cells of at least that size."""
    n = x.shape[0]
    cells = torch.clamp(torch.floor(length / reach), min=1).long()
    at = torch.minimum(torch.clamp(torch.floor((x - lo) / length * cells).long(), min=0), cells - 1)
    flat = (at[:, 2] * cells[1] + at[:, 1]) * cells[0] + at[:, 0]
    total = int(torch.prod(cells))
    order = torch.argsort(flat, stable=True)
    count = torch.bincount(flat, minlength=total)
    first = torch.cumsum(count, 0) - count
    table = torch.full((total, int(count.max())), n, dtype=torch.long, device=x.device)
    s = flat[order]
    table[s, torch.arange(n, device=x.device) - first[s]] = order
    xs = torch.cat([x, torch.full((1, 3), float("nan"), dtype=x.dtype, device=x.device)])  # no atom: never near
    around = [(-1, 0, 1) if int(k) >= 3 else (0, 1) if int(k) == 2 else (0,) for k in cells]
    ii, jj, sh = [], [], []
    for oz in around[2]:
        for oy in around[1]:
            for ox in around[0]:
                b = (at + torch.tensor([ox, oy, oz], device=x.device)) % cells
                cand = table[(b[:, 2] * cells[1] + b[:, 1]) * cells[0] + b[:, 0]]
                d = x[:, None, :] - xs[cand]
                image = torch.round(d / length)
                d = d - image * length
                near = ((d * d).sum(-1) <= reach * reach) & (cand != torch.arange(n, device=x.device)[:, None])
                i, k = torch.nonzero(near, as_tuple=True)
                ii.append(i)
                jj.append(cand[i, k])
                sh.append(image[i, k])
    return torch.cat(ii), torch.cat(jj), torch.cat(sh)


class _Lists:
    """The pairs of one list interval.  The reference refreshes ghosts pass by pass from values of
    the previous step, so an edge ghost lags its atom by one step and a corner ghost by two (never
    behind the list build); `lagged` False gives exact images."""

    def __init__(self, x, lo, length, reach, half, lagged):
        self.i, self.j, shift = _pairs(x, lo, length, reach)
        if half:
            keep = self.j < self.i
            self.i, self.j, shift = self.i[keep], self.j[keep], shift[keep]
        lag = torch.clamp((shift != 0).sum(-1) - 1, min=0) if lagged else torch.zeros_like(self.i)
        self.at = lag * x.shape[0] + self.j
        self.shift = shift * length
        self.half = half
        self.past = [x, x, x]

    def move(self, x):
        self.past = [x, self.past[0], self.past[1]]

    def delta(self):
        return self.past[0][self.i] - (torch.cat(self.past)[self.at] + self.shift)

    def gather(self, pair_force):
        f = torch.zeros_like(self.past[0]).index_add_(0, self.i, pair_force)
        return f.index_add_(0, self.j, -pair_force) if self.half else f


def _lj(lists, eps=1.0, sigma=1.0):
    """(forces, sums over the list's pairs inside the cutoff: energy, f r^2, number)."""
    d = lists.delta()
    r2 = (d * d).sum(-1)
    inside = r2 < LJ["cutoff"] ** 2
    sr2 = 1.0 / torch.where(inside, r2, torch.ones_like(r2))
    sr6 = sr2 ** 3 * sigma ** 6
    f = torch.where(inside, 48.0 * eps * sr6 * (sr6 - 0.5) * sr2, torch.zeros_like(r2))
    e = torch.where(inside, 4.0 * eps * sr6 * (sr6 - 1.0), torch.zeros_like(r2))
    return lists.gather(f[:, None] * d), (e.sum(), (f * r2).sum(), inside.sum().double())


def _dem(lists, v):
    """The contact model: overlap 2R - r, normal spring and dashpot, capped tangential dashpot."""
    dn, dtan, k, mu = DEM["params"]
    d = lists.delta()
    r2 = (d * d).sum(-1)
    touch = (r2 < min(DEM["cutoff"], 2 * DEM["radius"]) ** 2) & (r2 > 0)
    i, j, d, r = lists.i[touch], lists.j[touch], d[touch], torch.sqrt(r2[touch])
    n = d / r[:, None]
    rel = v[i] - v[j]
    vn = (rel * n).sum(-1)
    vt = rel - n * vn[:, None]
    speed = torch.sqrt((vt * vt).sum(-1))
    fn = torch.clamp(k * (2 * DEM["radius"] - r) - dn * vn, min=0.0)
    ft = torch.minimum(dtan * speed, mu * fn) / torch.where(speed > 0, speed, torch.ones_like(speed))
    return torch.zeros_like(v).index_add_(0, i, n * fn[:, None] - vt * ft[:, None])


def exact(c, seed):
    dev = _device()
    m, x, v, world, _ = _inputs(c, seed)
    if c["kind"] == "adjoint":
        x = tinymd.setup_particles("default", (c["nx"], c["ny"], c["nz"]), LATTICE)[1]
    lo = torch.tensor(world[0::2], device=dev)
    length = torch.tensor(world[1::2] - world[0::2], device=dev)
    x, v = torch.tensor(x, device=dev), torch.tensor(v, device=dev)
    if c["kind"] == "adjoint":
        return _exact_adjoint(c, x, v, lo, length, *_parameters(seed))
    model = _model(c)
    reach, dt = model["cutoff"] + SKIN, model["dt"]
    force = (lambda p, w: (_dem(p, w), None)) if model is DEM else (lambda p, w: _lj(p))
    lists = _Lists(x, lo, length, reach, c["half"], True)
    f, _ = force(lists, v)
    sums = []
    for k in range(c["steps"]):
        v = v + (0.5 * dt) * f
        x = x + dt * v
        if (k + 1) % REBUILD == 0:
            x = torch.where(x < lo, x + length, torch.where(x > lo + length, x - length, x))
            lists = _Lists(x, lo, length, reach, c["half"], True)
        else:
            lists.move(x)
        f, s = force(lists, v)
        v = v + (0.5 * dt) * f
        if c["kind"] == "monitor" and (k + 1) % READ_EVERY == 0:
            sums.append(torch.stack([*s, (v * v).sum()]))
    if c["kind"] == "evaluate":
        return [f]
    if c["form"] == "mixed":
        return [x, v]
    return [x, v, f] + ([torch.stack(sums)] if sums else [])


def _exact_adjoint(c, x, v, lo, length, eps, sigma):
    n, dt, reach = x.shape[0], LJ["dt"], LJ["cutoff"] + SKIN
    v0 = v.requires_grad_()
    eps = torch.tensor(eps, dtype=torch.float64, device=x.device, requires_grad=True)
    sigma = torch.tensor(sigma, dtype=torch.float64, device=x.device, requires_grad=True)

    def lists_at(y):
        wrapped = y.detach() - length * torch.floor((y.detach() - lo) / length)
        lists = _Lists(wrapped, lo, length, reach, False, False)
        # image shifts of the unwrapped positions
        d = y.detach()[lists.i] - y.detach()[lists.j]
        lists.shift = torch.round(d / length) * length
        lists.past = [y, y, y]
        return lists

    def one_step(lists, y, w, f, last):
        w = w + (0.5 * dt) * f
        y = y + dt * w
        if last:
            return y, w, f
        lists.move(y)
        f, _ = _lj(lists, eps, sigma)
        return y, w + (0.5 * dt) * f, f

    x0 = x
    lists = lists_at(x)
    f, _ = _lj(lists, eps, sigma)
    for k in range(c["steps"]):
        rebuild = (k + 1) % REBUILD == 0
        x, v, f = one_step(lists, x, v, f, rebuild)
        if rebuild:
            lists = lists_at(x)
            f, _ = _lj(lists, eps, sigma)
            v = v + (0.5 * dt) * f
    d = lists.delta()
    r2 = (d * d).sum(-1)
    inside = r2 < LJ["cutoff"] ** 2
    sr6 = sigma ** 6 / r2[inside] ** 3
    cut6 = (sigma / LJ["cutoff"]) ** 6
    energy = 0.5 * (4.0 * eps * (sr6 * (sr6 - 1.0) - cut6 * (cut6 - 1.0))).sum()
    loss = ((x - x0) ** 2).sum() / n + energy / n
    return [loss.detach(), *torch.autograd.grad(loss, [v0, eps, sigma])]
