"""The work a user has this framework do, as cases that can be timed and checked.

A case is one call that a program makes through the public entry points: a run of fused
Strang steps on one grid (``Grid.step``), a batch of independent solves (``Batch``), a
served mix (``Server``), or a multi-region propagation (``MultiRegionPropagator``).
Sizes, spacings, absorbers, potentials and pulses are those of the repository's own
configurations, benchmark and tests: 1D lines of 1024 .. 16384 points (any length), 2D
grids with edges 64 .. 2048, 3D cubes with edges 32 .. 256; both gauges, real time with
border fluxes and imaginary time with Normalize and the kinetic energy.  Everything is
complex128, the only type the path takes.

The start state is that of a run under way: a bound core and wave packets on their way
out, so that the fluxes, the absorber and the whole momentum range have something to do.
"""
import math

import numpy as np
import torch

import qsf_gb300 as Q
from qsf_gb300.multigrid import MultiGrid, MultiRegionPropagator
from qsf_gb300.serve import Server, grid_desc

DT_RE, DT_IM = 0.05, 0.01
DX = {1: 0.2, 2: 0.3, 3: 0.4}
EDGES = [64, 80, 96, 128, 160, 192, 256, 320, 384, 512, 640, 768, 1024, 1280, 1536, 2048]  # built 2D edges
CUBES = [32, 40, 48, 64, 80, 96, 128, 160, 192, 256]  # built 3D edges
BATCH_EDGES = [256, 384, 512, 768, 1024]
SERVE_EDGES = [256, 320, 384, 512]


def _grid_case(name, dim, n, steps, gauge="velocity", mode="real", absorber="cap", ekin_interval=0):
    return {"name": name, "kind": "grid", "dim": dim, "n": n, "steps": steps, "gauge": gauge, "mode": mode,
            "absorber": absorber, "ekin_interval": ekin_interval}


def listed():
    return [
        # the smallest call: a program that drives a short 1D line one step at a time
        _grid_case("line 1024, one step", 1, 1024, 1),
        # the 1D plain configuration: soft-core H, length gauge, cos^(1/8) mask, BOX flux
        _grid_case("line 4096, length gauge", 1, 4096, 256, gauge="length", absorber="cos8"),
        # a long served 1D solve: the line no longer fits one SM's shared memory
        _grid_case("line 12288", 1, 12288, 128),
        # a served 1D solve of an arbitrary length (the served 1D sizes are any integers)
        _grid_case("line 5003", 1, 5003, 64),
        # two electrons, a small grid run alone
        _grid_case("plane 384", 2, 384, 64),
        # two electrons, ground-state search: imaginary time, Normalize, E_kin every 10th step
        _grid_case("plane 1024, ground state", 2, 1024, 40, mode="imaginary", ekin_interval=10),
        # the 2D plain configuration (the headline workload): 2048^2, seven ZOA fluxes
        _grid_case("plane 2048", 2, 2048, 20),
        # the same physics on a grid edge outside 2^a, 3*2^a, 5*2^a
        _grid_case("plane 1000", 2, 1000, 16),
        # the 3D plain configuration: three electrons, length gauge, eight ZOA fluxes
        _grid_case("cube 256, length gauge", 3, 256, 8, gauge="length"),
        # a parameter scan: independent 2D solves of mixed edges advanced together
        {"name": "batch of 40", "kind": "batch", "solves": 40, "steps": 32},
        # a multi-region 2D grid (four regions, transfers and masks every step)
        {"name": "regions 1024", "kind": "regions", "dim": 2, "n": 1024, "omega": 3.0},
        # a burst of requests at the server: 1D lines of any length and 2D grids
        {"name": "served burst of 24", "kind": "serve", "requests": 24, "steps": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "plane", "plane", "plane", "cube", "batch", "regions", "serve"])
    gauge = rng.choice(["velocity", "length"])
    mode = rng.choice(["real", "real", "imaginary"])
    ek = rng.choice([0, 1, 10]) if mode == "imaginary" else 0
    if kind == "line":
        n = _log_int(rng, 256, 16384)
        if rng.random() < 0.6:  # a built length: 2^a, 3*2^a or 5*2^a
            n = min((q << a for q in (1, 3, 5) for a in range(6, 15) if q << a <= 16384), key=lambda v: abs(v - n))
        c = _grid_case("", 1, n, _log_int(rng, 1, 128), gauge, mode, rng.choice(["cap", "cos8"]), ek)
    elif kind == "plane":
        n = rng.choice(EDGES) if rng.random() < 0.7 else _log_int(rng, 63, 1000)
        most = max(1, min(64, 20 * 2048 * 2048 // (n * n * (1 if n in EDGES else 8))))
        c = _grid_case("", 2, n, _log_int(rng, max(1, most // 4), most), gauge, mode, "cap", ek)
    elif kind == "cube":
        n = rng.choice(CUBES)
        c = _grid_case("", 3, n, max(1, min(16, _log_int(rng, 2, 8) * 128 ** 3 // n ** 3)), gauge, mode, "cap", ek)
    elif kind == "batch":
        return {"kind": "batch", "solves": _log_int(rng, 6, 40), "steps": _log_int(rng, 8, 32)}
    elif kind == "regions":
        return {"kind": "regions", "dim": 2, "n": rng.choice([128, 192, 256, 320, 512, 768]),
                "omega": rng.choice([3.0, 4.0, 6.0])}
    else:
        return {"kind": "serve", "requests": _log_int(rng, 6, 24), "steps": _log_int(rng, 16, 64)}
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return np.random.default_rng(seed)


def _axis(n, dx):
    return torch.arange(n, dtype=torch.float64, device="cuda") * dx - 0.5 * dx * (n - 1)


def _state(dim, n, dx, rng):
    """Normalised psi: a bound core and four outgoing packets, on the GPU."""
    x = _axis(n, dx)
    half = 0.5 * n * dx
    psi = None
    for k in range(5):
        amp = 1.0 if k == 0 else rng.uniform(0.05, 0.3)
        f = None
        for _ in range(dim):
            w = 1.0 if k == 0 else rng.uniform(0.08, 0.2) * half
            c = 0.0 if k == 0 else rng.uniform(-0.5, 0.5) * half
            p = 0.0 if k == 0 else rng.uniform(-1.5, 1.5)
            line = torch.exp(-0.5 * ((x - c) / max(w, 1.0)) ** 2) * torch.exp(1j * p * x)
            f = line if f is None else f.unsqueeze(-1) * line
        psi = amp * f if psi is None else psi.add_(f, alpha=amp)
    return psi / math.sqrt(float(psi.abs().square().sum()) * dx ** dim)


def _pulse(dim, steps, gauge, rng):
    """Coupling rows of a sin^2 pulse under way: A per step (velocity gauge) or E at the
    opening and closing X half of each step (length gauge), the same on every axis."""
    amp = math.sqrt(10.0 ** rng.uniform(14.0, 15.0) / 3.50944e16)
    omega = 45.563352529 / rng.uniform(400.0, 1600.0)
    t0 = rng.uniform(0.2, 0.6) * 6.0 * math.pi / omega
    t = t0 + DT_RE * np.arange(steps + 1)
    e = amp * np.sin(omega * t) * np.sin(omega * t / 6.0) ** 2
    if gauge == "velocity":
        rows = np.zeros((steps, 3))
        rows[:, :dim] = (e[:-1] / omega)[:, None]
    else:
        rows = np.zeros((steps, 6))
        rows[:, :dim] = e[:-1, None]
        rows[:, 3:3 + dim] = e[1:, None]
    return rows


class _View:
    """psi of a grid as a device array, without a copy."""

    def __init__(self, grid):
        self.grid = grid
        self.__cuda_array_interface__ = {"shape": grid.shape, "typestr": "<c16", "version": 3,
                                         "data": (grid.device_ptr(), False)}


def _psi(grid):
    return torch.as_tensor(_View(grid), device="cuda")


def _grid_args(case):
    """What Grid takes for a grid case, and the observables of its steps."""
    dim, n = case["dim"], case["n"]
    real = case["mode"] == "real"
    ncap = max(1, n // 10)
    args = dict(dim=dim, n=n, dx=DX[dim], nCAP=ncap, Ncharge=float(dim),
                gauge=Q.GAUGE_LENGTH if case["gauge"] == "length" else Q.GAUGE_VELOCITY, n_fields=1 if real else 0)
    if case["absorber"] == "cos8":
        args.update(absorber=Q.ABS_COS8, mask_dt=DT_RE if real else DT_IM)
    obs = Q.OBS_NORM | Q.OBS_EPOT
    step = dict(mode=Q.MODE_RE if real else Q.MODE_IM, dt=DT_RE if real else DT_IM, nsteps=case["steps"])
    if case["ekin_interval"]:
        obs |= Q.OBS_EKIN
        step["ekin_interval"] = case["ekin_interval"]
    if not real:
        step["normalize"] = True
    elif dim == 1:
        step.update(borders=["BOX"], box_size=max(4, (2 * n) // 5 - 2))
    else:
        step["borders"] = Q.ZOA_FLUX_2D if dim == 2 else Q.ZOA_FLUX_3D
    step["obs"] = obs
    return args, step


def _border_nodes(n):
    """The default border distances, drawn in on grids too small for them."""
    return (25, 14, 10, 40) if n >= 128 else (max(3, n // 6), max(2, n // 10), max(2, n // 12), max(4, n // 4))


def _batch_specs(case, rng):
    edges = rng.choice(BATCH_EDGES, case["solves"])
    edges[:2] = BATCH_EDGES[0], BATCH_EDGES[-1]
    return [int(e) for e in edges]


def _serve_specs(case, rng):
    """(dim, n) per request: half 1D lines of any length, half 2D grids."""
    out = []
    for k in range(case["requests"]):
        out.append((1, int(rng.integers(1024, 16385))) if k % 2 else (2, int(rng.choice(SERVE_EDGES))))
    return out


SIZES_SEED = 20  # a batch's and a burst's sizes belong to the case, their inputs to the seed


def prepare(case, seed):
    rng = _gen(seed)
    if case["kind"] == "grid":
        args, step = _grid_args(case)
        grid = Q.Grid(border_nodes=_border_nodes(case["n"]), **args)
        psi0 = _state(case["dim"], case["n"], args["dx"], rng)
        _psi(grid).copy_(psi0)
        if case["mode"] == "real":
            step["coupling"] = _pulse(case["dim"], case["steps"], case["gauge"], rng)
        torch.cuda.synchronize()
        return {"case": case, "grid": grid, "step": step, "psi": _psi(grid)}
    if case["kind"] == "batch":
        members = []
        for e in _batch_specs(case, _gen(SIZES_SEED)):
            g = Q.Grid(2, e, DX[2], nCAP=e // 10, Ncharge=2.0, gauge=Q.GAUGE_VELOCITY, n_fields=1)
            _psi(g).copy_(_state(2, e, DX[2], rng))
            members.append((g, _pulse(2, case["steps"], "velocity", rng), _psi(g)))
        torch.cuda.synchronize()
        return {"case": case, "batch": Q.Batch(), "members": members}
    if case["kind"] == "regions":
        mg = MultiGrid(2, case["n"], DX[2], case["n"] // 10, Ncharge=2.0, gauge=Q.GAUGE_VELOCITY, n_fields=1)
        psis = [_psi(g) for g in mg.regions]
        psis[0].copy_(_state(2, case["n"], DX[2], rng))
        torch.cuda.synchronize()
        amp = math.sqrt(10.0 ** rng.uniform(14.0, 15.0) / 3.50944e16)
        return {"case": case, "mg": mg, "psis": psis, "amp": amp}
    reqs = []
    for dim, n in _serve_specs(case, _gen(SIZES_SEED)):
        d = grid_desc(dim, n, DX[dim], nCAP=n // 10, Ncharge=float(dim), gauge=Q.GAUGE_VELOCITY, n_fields=1)
        kw = dict(borders=["BOX"], box_size=(2 * n) // 5) if dim == 1 else dict(borders=Q.ZOA_FLUX_2D)
        reqs.append((d, _pulse(dim, case["steps"], "velocity", rng), _state(dim, n, DX[dim], rng).cpu().numpy(), kw))
    return {"case": case, "server": Server(max_slots=32, steps_per_round=16), "reqs": reqs}


# ------------------------------------------------------------------ one call
def _columns(rows):
    return {"norm": rows[..., 0], "epot": rows[..., 1], "ekin": rows[..., 2], "flux": rows[..., 3:]}


def run(state):
    case = state["case"]
    if case["kind"] == "grid":
        rows, done = state["grid"].step(**state["step"])
        return {"psi": state["psi"], "done": done, **_columns(rows)}
    if case["kind"] == "batch":
        b, steps = state["batch"], case["steps"]
        slots = [b.add(g, Q.MODE_RE, DT_RE, steps, pulse, obs=Q.OBS_NORM | Q.OBS_EPOT, borders=Q.ZOA_FLUX_2D)
                 for g, pulse, _ in state["members"]]
        b.run(steps)
        rows = np.stack([b.result(s)[0] for s in slots])
        for s in slots:
            b.remove(s)
        return {"psi": [psi for _, _, psi in state["members"]], **_columns(rows)}
    if case["kind"] == "regions":
        mg = state["mg"]
        pulse = Q.Pulse(field=state["amp"], omega=case["omega"], ncycles=1.0)
        prop = MultiRegionPropagator(DT_RE, mg, Q.Coupling(Q.GAUGE_VELOCITY, [Q.Field(3, [pulse])]), ["norm", "epot"])
        rows = prop.run()
        return {"psi": state["psis"], "norm": np.array([r["norm"] for r in rows]),
                "epot": np.array([r["epot"] for r in rows])}
    srv = state["server"]
    tickets = [srv.submit(d, Q.MODE_RE, DT_RE, case["steps"], pulse, psi0, obs=Q.OBS_NORM | Q.OBS_EPOT, **kw)
               for d, pulse, psi0, kw in state["reqs"]]
    res = [srv.wait(t) for t in tickets]
    return {"norm": np.array([r["final_norm"] for r in res]), "epot": np.array([r["final_epot"] for r in res]),
            "flux": np.array([r["flux_integral"][:len(Q.ZOA_FLUX_2D)] for r in res]),
            "status": np.array([r["status"] for r in res]), "steps": np.array([r["steps"] for r in res])}


# ------------------------------------------------------------------ what it cannot do without
def _grid_work(dim, n, steps, ekin=0):
    """psi in and out once; per step the forward and inverse transform (5 n log2 n each),
    three phase products, norm and potential energy; a further transform per E_kin."""
    m = float(n) ** dim
    fft = 5.0 * m * math.log2(m)
    return np.array([32.0 * m, steps * (2.0 * fft + 26.0 * m) + ekin * (fft + 5.0 * m)])


def work(case):
    if case["kind"] == "grid":
        k = case["ekin_interval"]
        w = _grid_work(case["dim"], case["n"], case["steps"], -(-case["steps"] // k) if k else 0)
    elif case["kind"] == "batch":
        w = sum(_grid_work(2, e, case["steps"]) for e in _batch_specs(case, _gen(SIZES_SEED)))
    elif case["kind"] == "regions":
        steps = int(2.0 * math.pi / case["omega"] / DT_RE) + 3
        w = 4 * _grid_work(2, case["n"], steps)
    else:
        w = sum(_grid_work(d, n, case["steps"]) for d, n in _serve_specs(case, _gen(SIZES_SEED)))
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ------------------------------------------------------------------ the same in plain torch
def _broadcast(v, d, dim):
    return v.reshape([-1 if k == d else 1 for k in range(dim)])


def _exact_steps(psi, dim, n, dx, steps, mode, gauge, absorber, rows, ekin_interval, normalize):
    x = _axis(n, dx)
    idx = torch.arange(n, device="cuda")
    k = torch.where(idx < n // 2, idx, idx - n).double() * (2.0 * math.pi / n / dx)
    ncap, dt = max(1, n // 10), DT_RE if mode == "real" else DT_IM
    unit = -1j if mode == "real" else -1.0
    one = [_broadcast(x, d, dim) for d in range(dim)]
    V = sum(-float(dim) / torch.sqrt(c * c + 1.0) for c in one)
    for a in range(dim):
        for b in range(a):
            V = V + 1.0 / torch.sqrt((one[a] - one[b]) ** 2 + 1.0)
    node = (ncap + torch.where(idx < n // 2, -idx, idx - n + 1)).clamp(min=0).double()
    if absorber == "cap":
        damp = -0.5 * dt * node ** 4 * (3.0 / ncap) ** 4
    else:
        damp = 0.5 * 0.125 * torch.log(torch.cos(0.5 * math.pi * node / ncap))
    X = torch.exp(unit * 0.5 * dt * V + sum(_broadcast(damp, d, dim) for d in range(dim)))
    dV = dx ** dim
    axes = list(range(dim))
    K2 = sum(_broadcast(0.5 * k * k, d, dim) for d in range(dim))
    out = {"norm": [], "epot": [], "ekin": []}

    def half(f, e):
        f = f * X
        if gauge == "length" and rows is not None:
            for d in range(dim):
                f = f * _broadcast(torch.exp(unit * 0.5 * dt * float(e[d]) * x), d, dim)
        return f

    for s in range(steps):
        A = rows[s] if rows is not None and gauge == "velocity" else np.zeros(3)
        psi = half(psi, rows[s][:3] if rows is not None and gauge == "length" else None)
        psi = torch.fft.fftn(psi, dim=axes)
        for d in range(dim):
            psi = psi * _broadcast(torch.exp(unit * dt * (0.5 * k * k + k * float(A[d]))), d, dim)
        psi = torch.fft.ifftn(psi, dim=axes)
        psi = half(psi, rows[s][3:] if rows is not None and gauge == "length" else None)
        rho = psi.abs().square()
        nrm = float(rho.sum()) * dV
        out["norm"].append(nrm)
        out["epot"].append(float((rho * V).sum()) * dV)
        ek = ekin_interval and ((s + 1) % ekin_interval == 0 or s + 1 == steps)
        out["ekin"].append(float((torch.fft.fftn(psi, dim=axes).abs().square() * K2).sum()) * dV / float(n) ** dim
                           if ek else 0.0)
        if normalize:
            psi = psi * math.sqrt(1.0 / nrm)
    return psi, {c: np.array(v) for c, v in out.items()}


def exact(case, seed):
    """The fluxes have no value here: their borders are a table of this framework's own."""
    rng = _gen(seed)
    if case["kind"] == "grid":
        dim, n, real = case["dim"], case["n"], case["mode"] == "real"
        psi = _state(dim, n, DX[dim], rng)
        rows = _pulse(dim, case["steps"], case["gauge"], rng) if real else None
        psi, cols = _exact_steps(psi, dim, n, DX[dim], case["steps"], case["mode"], case["gauge"], case["absorber"], rows,
                                 case["ekin_interval"], not real)
        return {"psi": psi, "done": case["steps"], "flux": None, **cols}
    if case["kind"] == "regions":
        return None  # the transfers between regions are this framework's own definition
    if case["kind"] == "batch":
        sizes = [(2, e) for e in _batch_specs(case, _gen(SIZES_SEED))]
    else:
        sizes = _serve_specs(case, _gen(SIZES_SEED))
    psis, cols = [], []
    for dim, n in sizes:
        if case["kind"] == "batch":
            psi = _state(dim, n, DX[dim], rng)
            rows = _pulse(dim, case["steps"], "velocity", rng)
        else:
            rows = _pulse(dim, case["steps"], "velocity", rng)
            psi = _state(dim, n, DX[dim], rng)
        psi, c = _exact_steps(psi, dim, n, DX[dim], case["steps"], "real", "velocity", "cap", rows, 0, False)
        psis.append(psi)
        cols.append(c)
    if case["kind"] == "batch":
        return {"psi": psis, "flux": None, **{k: np.stack([c[k] for c in cols]) for k in ("norm", "epot", "ekin")}}
    return {"norm": np.array([c["norm"][-1] for c in cols]), "epot": np.array([c["epot"][-1] for c in cols]),
            "flux": None, "status": np.zeros(len(cols), dtype=np.int64),
            "steps": np.full(len(cols), case["steps"], dtype=np.int64)}
