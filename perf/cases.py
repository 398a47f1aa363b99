"""The work that users of this framework have it do, as timed cases.

A case is one call sequence a program makes: a lattice brought to a state,
stepped for a report interval and read back; a batch of lattices stepped
together; a set of lattices compared as the precision sweep compares them; a
set of requests served.  `listed` names fixed ones, `draw` picks more from the
same ranges, `prepare` makes what a program holds before the call, `run` is
the call, `work` what it cannot do without and `exact` its float64 result in
plain torch.
"""
import math
import time

import numpy as np
import torch

import imexlbm_gb300 as imex
from imexlbm_gb300 import LBM, Batch, Server

PREC = {"f64": imex.IMEX_F64, "f32": imex.IMEX_F32, "f16": imex.IMEX_F16DEV}
PI = 3.1415926  # the reference's value, in tau and in the initial field


def listed():
    return [
        # the reference's regression-size deck: 32^3, reported every 10 steps
        # as its main loop does (the smallest lattice anyone runs alone)
        {"name": "deck32_f64", "kind": "deck", "nx": 32, "ny": 32, "nz": 32, "precision": "f64", "steps": 100,
         "every": 10},
        # the shipped deck's lattice, float64, from a given state to the next report
        {"name": "shipped256_f64", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "precision": "f64",
         "rounding": "nearest", "steps": 20},
        # float64 on a ragged box, as decks with three different sizes give
        {"name": "ragged_f64", "kind": "solve", "nx": 90, "ny": 77, "nz": 131, "precision": "f64",
         "rounding": "nearest", "steps": 40},
        # the shipped lattice in float32 storage
        {"name": "shipped256_f32", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "precision": "f32",
         "rounding": "nearest", "steps": 40},
        # float32, ragged and odd
        {"name": "ragged_f32", "kind": "solve", "nx": 121, "ny": 150, "nz": 97, "precision": "f32",
         "rounding": "nearest", "steps": 60},
        # the shipped lattice as float16 deviations with the default (stochastic) rounding
        {"name": "shipped256_f16", "kind": "solve", "nx": 256, "ny": 256, "nz": 256, "precision": "f16",
         "rounding": "stochastic", "steps": 40},
        # float16 deviations rounded to nearest, ragged and odd
        {"name": "ragged_f16", "kind": "solve", "nx": 84, "ny": 99, "nz": 107, "precision": "f16",
         "rounding": "nearest", "steps": 60},
        # a small float32 solve alone, the most frequent kind of size in the served mix
        {"name": "small64_f32", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "precision": "f32",
         "rounding": "nearest", "steps": 200},
        # many float32 lattices of uneven edges in one batch (the batched workload's range)
        {"name": "batch_f32", "kind": "batch", "members": 24, "edge_min": 32, "edge_max": 128, "mix": 0.0,
         "multiple": 16, "steps": 96},
        # a batch of both formats with edges of any parity (the served workload's range)
        {"name": "batch_mixed", "kind": "batch", "members": 24, "edge_min": 24, "edge_max": 160, "mix": 0.5,
         "multiple": 1, "steps": 64},
        # one report of the precision sweep: float64, float32 and float16 lattices compared
        {"name": "sweep128", "kind": "sweep", "nx": 128, "ny": 128, "nz": 128, "steps": 40},
        # a burst of requests served from submission to the last result
        {"name": "served_burst", "kind": "served", "members": 24, "edge_min": 32, "edge_max": 128, "mix": 0.5,
         "steps": 300},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("deck", "solve", "solve", "solve", "solve", "batch", "batch", "sweep", "served"))
    if kind == "deck":
        c = {"kind": kind, "precision": "f64", "every": rng.choice((5, 10, 20))}
        c["nx"], c["ny"], c["nz"] = (_log_int(rng, 12, 64) for _ in range(3))
        c["steps"] = c["every"] * rng.randint(4, 10)
        return c
    if kind == "solve":
        prec = rng.choice(("f64", "f32", "f16"))
        rounding = rng.choice(("stochastic", "nearest")) if prec == "f16" else "nearest"
        c = {"kind": kind, "precision": prec, "rounding": rounding}
        c["nx"], c["ny"], c["nz"] = (_log_int(rng, 20, 256) for _ in range(3))
        if rng.random() < 0.4:  # aligned rows, as most decks have
            c["nz"] = max(16, c["nz"] // 16 * 16)
        cells = c["nx"] * c["ny"] * c["nz"]
        c["steps"] = max(3, min(rng.randint(20, 200), int(3.0e8 / cells) if prec == "f64" else int(6.0e8 / cells)))
        return c
    if kind == "batch":
        lo = _log_int(rng, 16, 64)
        return {"kind": kind, "members": rng.randint(4, 28), "edge_min": lo,
                "edge_max": min(144, _log_int(rng, 2 * lo, 4 * lo)), "mix": rng.choice((0.0, 0.5, 1.0)),
                "multiple": rng.choice((1, 8, 16)), "steps": rng.randint(17, 64)}
    if kind == "sweep":
        c = {"kind": kind, "steps": rng.randint(10, 40)}
        c["nx"], c["ny"], c["nz"] = (_log_int(rng, 32, 128) for _ in range(3))
        return c
    return {"kind": "served", "members": rng.randint(8, 24), "edge_min": 32, "edge_max": rng.choice((64, 96, 128)),
            "mix": rng.choice((0.0, 0.5, 1.0)), "steps": rng.randint(100, 300)}


# ------------------------------------------------------------------ inputs --
def _tau(u0, nx, re):
    return u0 * nx / re / (1.0 / 3.0) / 2.0 / PI


def _flow(rng, nx):
    """A Taylor-Green flow: u0, Re, phase and the relaxation time."""
    u0 = float(rng.uniform(0.02, 0.08))
    re = int(round(math.exp(rng.uniform(math.log(100), math.log(1600)))))
    return {"u0": u0, "tau": _tau(u0, nx, re), "phase": [float(x) for x in rng.uniform(0.0, 2 * math.pi, 3)]}


def _members(case, seed):
    """The lattices of a batch or the requests of a burst: edges spread over
    the case's range (the same for every seed: the workload's shape), the
    flows from the seed."""
    rng = np.random.default_rng([int(seed), 7])
    n, lo, hi = case["members"], case["edge_min"], case["edge_max"]
    mult = case.get("multiple", 32)
    out = []
    for i in range(n):
        edge = lo * (hi / lo) ** (((i * 11) % n) / max(1, n - 1))
        edge = max(mult, int(round(edge / mult)) * mult) if mult > 1 else int(round(edge))
        m = _flow(rng, edge)
        m["edge"] = edge
        m["precision"] = "f16" if ((i * 7) % n + 0.5) / n < case["mix"] else "f32"
        m["steps"] = max(1, int(round(case["steps"] * (0.4 + 0.6 * (((i * 5) % n) / max(1, n - 1))))))
        out.append(m)
    return out


def _axis(n, shift):
    return torch.arange(n, dtype=torch.float64, device="cuda") / n * 2.0 * PI + shift


def _directions():
    pairs = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1),
             (1, 1, 1), (1, -1, 1), (1, 1, -1), (1, -1, -1)]
    e = [(0, 0, 0)]
    for p in pairs:
        e += [p, tuple(-c for c in p)]
    w = [(8 / 27, 2 / 27, 1 / 54, 1 / 216)[sum(c != 0 for c in d)] for d in e]
    return e, w


def _equilibrium(s, u, v, w):
    """w_a (s + 3 e.u + 4.5 (e.u)^2 - 1.5 u.u) of fields s = 3p, u, v, w."""
    e, wt = _directions()
    base = s - 1.5 * (u * u + v * v + w * w)
    f = torch.empty((27,) + tuple(s.shape), dtype=torch.float64, device="cuda")
    for a in range(27):
        edu = e[a][0] * u + e[a][1] * v + e[a][2] * w
        f[a] = wt[a] * (base + 3.0 * edu + 4.5 * edu * edu)
    return f


def _taylor_green(nx, ny, nz, u0, phase, rho0=1.0):
    x = _axis(nx, phase[0])[:, None, None]
    y = _axis(ny, phase[1])[None, :, None]
    z = _axis(nz, phase[2])[None, None, :]
    u = u0 * torch.sin(x) * torch.cos(y) * torch.cos(z)
    v = -u0 * torch.cos(x) * torch.sin(y) * torch.cos(z)
    p = rho0 / 3.0 + rho0 * u0 * u0 / 16.0 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)
    return _equilibrium(3.0 * p, u, v, torch.zeros_like(u))


def _lattice(nx, ny, nz, precision, flow, rounding=None):
    lat = LBM(nx, ny, nz, flow["tau"], 1.0, flow["u0"], precision=PREC[precision])
    if precision == "f16" and rounding is not None:
        lat.set_rounding(imex.IMEX_ROUND_STOCHASTIC if rounding == "stochastic" else imex.IMEX_ROUND_NEAREST)
    return lat


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "served"):
        members = _members(case, seed)
        if kind == "served":
            return {"case": case, "members": members, "server": Server(60e9, 64, 25)}
        lats = [_lattice(m["edge"], m["edge"], m["edge"], m["precision"], m) for m in members]
        batch = Batch(64)
        for m, lat in zip(members, lats):
            lat.initialize_phase(*m["phase"])
            batch.add(lat)
        out = torch.empty(27 * sum(m["edge"] ** 3 for m in members), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return {"case": case, "members": members, "lats": lats, "batch": batch, "out": out}
    shape = (case["nx"], case["ny"], case["nz"])
    flow = _flow(np.random.default_rng([int(seed), 3]), shape[0])
    state = {"case": case, "flow": flow}
    if kind == "sweep":
        state["lats"] = [_lattice(*shape, p, flow) for p in ("f64", "f32", "f16")]
        state["out"] = torch.empty((3, 27) + shape, dtype=torch.float64, device="cuda")
    else:
        state["lat"] = _lattice(*shape, case["precision"], flow, case.get("rounding"))
        state["out"] = torch.empty((27,) + shape, dtype=torch.float64, device="cuda")
    if kind == "solve":
        state["f0"] = _taylor_green(*shape, flow["u0"], flow["phase"])
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "deck":
        lat, out = state["lat"], state["out"]
        lat.initialize_phase(*state["flow"]["phase"])
        cons = []
        for _ in range(steps // case["every"]):
            lat.step(case["every"])
            cons.append(lat.Conserved())
        lat.get_f_device(out.data_ptr(), out.numel())
        return {"f": out, "conserved": np.array(cons)}
    if kind == "solve":
        lat, f0, out = state["lat"], state["f0"], state["out"]
        lat.set_f_device(f0.data_ptr(), f0.numel())
        lat.step(steps)
        cons = lat.Conserved()
        lat.get_f_device(out.data_ptr(), out.numel())
        return {"f": out, "conserved": np.array(cons)}
    if kind == "sweep":
        lats, out = state["lats"], state["out"]
        for lat in lats:
            lat.initialize_phase(*state["flow"]["phase"])
            lat.step(steps)
        diffs = [lat.velocity_max_diff(lats[0]) for lat in lats[1:]]
        cons = [lat.Conserved() for lat in lats]
        ranges = [lat.minmax_uvwp() for lat in lats]
        for lat, o in zip(lats, out):
            lat.get_f_device(o.data_ptr(), o.numel())
        return {"f": out, "conserved": np.array(cons), "ranges": np.array(ranges), "differences": np.array(diffs)}
    if kind == "batch":
        out, at = state["out"], 0
        for m, lat in zip(state["members"], state["lats"]):
            lat.initialize_phase(*m["phase"])
        state["batch"].step(steps)
        state["batch"].synchronize()
        cons = []
        for lat in state["lats"]:
            n = 27 * lat.glx * lat.gly * lat.glz
            cons.append(lat.Conserved())
            lat.get_f_device(out.data_ptr() + 8 * at, n)
            at += n
        return {"f": out, "conserved": np.array(cons)}
    server, members = state["server"], state["members"]
    for i, m in enumerate(members):
        server.submit(m["edge"], m["edge"], m["edge"], m["tau"], m["u0"], m["steps"], PREC[m["precision"]],
                      phase=m["phase"], tag=i)
    done = {}
    while len(done) < len(members):
        for r in server.poll():
            done[r["tag"]] = r
        time.sleep(0.0005)
    return {"conserved": np.array([done[i]["conserved"] for i in range(len(members))]),
            "steps": np.array([done[i]["steps"] for i in range(len(members))])}


# -------------------------------------------------------------------- work --
def _updates(case):
    if case["kind"] in ("batch", "served"):
        ms = _members(case, 0)
        cells = [m["edge"] ** 3 for m in ms]
        if case["kind"] == "batch":
            return sum(cells), sum(cells) * case["steps"]
        return sum(cells), sum(c * m["steps"] for c, m in zip(cells, ms))
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "sweep":
        return 3 * cells, 3 * cells * case["steps"]
    return cells, cells * case["steps"]


def work(case):
    """The float64 state given (where one is) read once and the one asked for
    written once, 216 bytes a cell each; 594 operations a cell and step, the
    reference's own count of its collision and streaming."""
    cells, updates = _updates(case)
    sides = {"solve": 2, "served": 0}.get(case["kind"], 1)
    return {"bytes": 27 * 8 * cells * sides, "flops": 594 * updates}


# ------------------------------------------------------------------- exact --
def _evolve(f, tau, steps, every=None):
    """`steps` float64 time steps (collide, then stream) and the conserved
    sums every `every` steps."""
    e, wt = _directions()
    omega = 1.0 / (tau + 0.5)
    cons = []
    for n in range(1, steps + 1):
        s, u, v, w = _moments(f)
        base = s - 1.5 * (u * u + v * v + w * w)
        for a in range(27):
            edu = e[a][0] * u + e[a][1] * v + e[a][2] * w
            c = f[a] + omega * (wt[a] * (base + 3.0 * edu + 4.5 * edu * edu) - f[a])
            f[a] = torch.roll(c, e[a], dims=(0, 1, 2)) if a else c
        if every and n % every == 0:
            cons.append(_conserved(f))
    return f, cons


def _moments(f):
    e, _ = _directions()
    m = [torch.zeros_like(f[0]) for _ in range(4)]
    for a in range(27):
        m[0] += f[a]
        for d in range(3):
            if e[a][d]:
                m[d + 1] += e[a][d] * f[a]
    return m


def _conserved(f):
    s, u, v, w = _moments(f)
    return [float(x.sum()) for x in (s, u, v, w)] + [float(0.5 * (u * u + v * v + w * w).sum())]


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind in ("batch", "served"):
        fs, cons, counts = [], [], []
        for m in _members(case, seed):
            n = steps if kind == "batch" else m["steps"]
            f, _ = _evolve(_taylor_green(m["edge"], m["edge"], m["edge"], m["u0"], m["phase"]), m["tau"], n)
            cons.append(_conserved(f))
            counts.append(n)
            if kind == "batch":
                fs.append(f.reshape(-1))
        if kind == "served":
            return {"conserved": np.array(cons), "steps": np.array(counts)}
        return {"f": torch.cat(fs), "conserved": np.array(cons)}
    shape = (case["nx"], case["ny"], case["nz"])
    flow = _flow(np.random.default_rng([int(seed), 3]), shape[0])
    f = _taylor_green(*shape, flow["u0"], flow["phase"])
    f, cons = _evolve(f, flow["tau"], steps, case.get("every"))
    if kind == "sweep":
        s, u, v, w = _moments(f)
        r = [float(x.max()) for x in (u, v, w, s / 3.0)] + [float(x.min()) for x in (u, v, w, s / 3.0)]
        return {"f": f.expand(3, *f.shape), "conserved": np.array([_conserved(f)] * 3), "ranges": np.array([r] * 3),
                "differences": None}
    return {"f": f, "conserved": np.array(cons if kind == "deck" else _conserved(f))}
