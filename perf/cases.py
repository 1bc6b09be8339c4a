"""Timed cases: the work users of this engine have it do, through its public
entry points.

    listed()             the cases that are always measured
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call
    run(state)           one pass; returns the outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the outputs of one pass in 64-bit torch, without the engine

Four kinds of pass:

  steps     n velocity-Verlet steps of a resident system (the solver's
            `solve` loop), NVE or coupled, and the state back on the host;
            "upload" cases bring fresh host arrays and the initial forces into
            the pass as well
  ensemble  n steps of many independent replicas on one device
  frame     one saved frame: upload, forces, macro parameters of every type
            (the CLI's `solve-macro-parameters` loop)
  render    the headless picture of a frame

Sizes, state points, couplings and units are those of the configurations the
benchmark runs (argon in nm/ps/K units; LJ liquids in reduced units at rho* =
0.8442, T* = 0.72), with odd and ragged sizes between them.  Threads per atom
are fixed wherever the engine would otherwise choose them by timing, as a
program does that wants the same bits from run to run.
"""
import math

import numpy as np
import torch

from moldyn_gb300 import render as rnd
from moldyn_gb300.core import ParticleDatabase, State
from moldyn_gb300.engine import Engine
from moldyn_gb300.initializer import Barostat, Thermostat
from moldyn_gb300.solver import Integrator, Potential, PotentialsDatabase

K_B = 1.380648528
RHO, T_STAR, DT, SKIN = 0.8442, 0.72, 0.005, 0.3
ARGON = {"edge": 3.338339, "mass": 66.335, "radius": 0.071, "sigma": 0.3405, "eps": 119.8 * K_B * 0.01}
# (type, type) -> (sigma, eps) of the two-type systems, and their masses
MIX = {(0, 0): (1.0, 1.0), (0, 1): (0.95, 0.9), (1, 1): (0.9, 0.8)}
MIX_MASS = (1.0, 2.0)


def _steps(name, system, nx, ny, nz, steps, precision, reference_order=False, coupling="nve", api="engine",
           graph_steps=0, threads_per_atom=1, frame_every=0, upload=False):
    return {"name": name, "kind": "steps", "system": system, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "precision": precision, "reference_order": reference_order, "coupling": coupling, "api": api,
            "graph_steps": graph_steps, "threads_per_atom": threads_per_atom,
            "frame_every": frame_every or steps, "upload": upload}


def _frame(name, nx, ny, nz, precision, reference_order, types=1, threads_per_atom=1):
    return {"name": name, "kind": "frame", "system": "liquid", "nx": nx, "ny": ny, "nz": nz, "types": types,
            "precision": precision, "reference_order": reference_order, "threads_per_atom": threads_per_atom}


def _ensemble(name, nrep, sizes_seed, steps, threads_per_atom=1):
    return {"name": name, "kind": "ensemble", "nrep": nrep, "sizes_seed": sizes_seed, "steps": steps,
            "threads_per_atom": threads_per_atom}


def _render(name, nx, ny, nz, width, height, mode):
    return {"name": name, "kind": "render", "nx": nx, "ny": ny, "nz": nz, "width": width, "height": height,
            "mode": mode}


def listed():
    return [
        # the solver crate's own call, one step a call, on the argon example:
        # the smallest thing a user does, all latency
        _steps("argon_1k_calculate", "argon", 10, 10, 10, 1, "fp64", True, "berendsen", api="calculate"),
        # the same system as `solve` runs it with --frames-per-save 100, at the
        # CLI's default precision (FP64 in the reference's summation order)
        _steps("argon_1k_solve_fp64", "argon", 10, 10, 10, 100, "fp64", True, "berendsen"),
        # a small liquid on the mixed path: equilibration runs, parameter scans
        _steps("liquid_2k_mixed", "liquid", 7, 8, 9, 100, "mixed"),
        # `solve` with its default of a saved frame per step, on a ragged
        # mid-size box at the CLI's default precision
        _steps("liquid_23k_solve_fp64", "liquid", 17, 18, 19, 10, "fp64", True, frame_every=1),
        # a thermostatted mid-size run on the mixed path
        _steps("liquid_55k_nose_hoover", "liquid", 23, 24, 25, 50, "mixed", coupling="nose_hoover",
               threads_per_atom=2),
        # the drift study's plain FP64 leg
        _steps("liquid_256k_fp64", "liquid", 40, 40, 40, 20, "fp64"),
        # the headline workload end to end: host arrays up, initial forces, 20
        # NVE steps, the whole state back
        _steps("liquid_1m_end_to_end", "liquid", 50, 50, 100, 20, "mixed", graph_steps=64, upload=True),
        # the large box with both Berendsen couplings
        _steps("liquid_8m_berendsen", "liquid", 100, 100, 200, 20, "mixed", coupling="berendsen"),
        # the uneven ensemble: one persistent launch per force pass, one graph of 50 steps
        _ensemble("ensemble_512", 512, 2024, 50),
        # analysis of saved frames at the CLI's default precision ...
        _frame("frame_110k_macro_fp64", 29, 30, 32, "fp64", True),
        # ... and of a two-type mixture on the mixed path
        _frame("frame_mixture_500k", 50, 50, 51, "mixed", False, types=2),
        # the viewer's picture of the headline box at full HD
        _render("render_1m_1080p", 50, 50, 100, 1920, 1080, "speed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, lo, hi):
    """Three FCC edge lengths whose product is log-uniform in lo .. hi cells."""
    edge = math.exp(rng.uniform(math.log(lo), math.log(hi)) / 3.0)
    return tuple(max(4, int(round(edge * rng.uniform(0.85, 1.18)))) for _ in range(3))


def draw(rng):
    what = rng.choice(["argon", "small", "solve", "mid", "fp64", "large", "coupled", "ensemble", "frame", "mixture",
                       "render"])
    c = None
    if what == "argon":
        e = [rng.randint(7, 14) for _ in range(3)]
        api = rng.choice(["calculate", "engine"])
        c = _steps("", "argon", *e, 1 if api == "calculate" else rng.randint(20, 120), "fp64", True,
                   rng.choice(["berendsen", "nve"]), api=api)
    elif what == "small":
        c = _steps("", "liquid", *_cells(rng, 200, 4000), rng.randint(20, 120), "mixed",
                   coupling=rng.choice(["nve", "berendsen", "nose_hoover"]))
    elif what == "solve":
        k = rng.randint(2, 10)
        c = _steps("", "liquid", *_cells(rng, 500, 12000), k, "fp64", True,
                   coupling=rng.choice(["nve", "berendsen"]), frame_every=rng.choice([1, k]))
    elif what == "mid":
        c = _steps("", "liquid", *_cells(rng, 4000, 64000), rng.randint(10, 60), "mixed",
                   coupling=rng.choice(["nve", "berendsen", "nose_hoover"]), threads_per_atom=rng.choice([1, 2]),
                   graph_steps=rng.choice([0, 32]))
    elif what == "fp64":
        c = _steps("", "liquid", *_cells(rng, 8000, 100000), rng.randint(5, 20), "fp64",
                   coupling=rng.choice(["nve", "berendsen"]))
    elif what == "large":
        c = _steps("", "liquid", *_cells(rng, 100000, 700000), rng.randint(10, 30), "mixed", graph_steps=64,
                   upload=rng.choice([True, False]))
    elif what == "coupled":
        c = _steps("", "liquid", *_cells(rng, 100000, 1000000), rng.randint(5, 20), "mixed", coupling="berendsen")
    elif what == "ensemble":
        c = _ensemble("", _log_int(rng, 16, 400), rng.randint(1, 10 ** 6), rng.randint(10, 50))
    elif what == "frame":
        ref = rng.random() < 0.5
        c = _frame("", *_cells(rng, 500, 40000 if ref else 300000), "fp64" if ref else "mixed", ref)
    elif what == "mixture":
        c = _frame("", *_cells(rng, 500, 150000), "mixed", False, types=2)
    else:
        w = rng.randint(320, 2560)
        c = _render("", *_cells(rng, 300, 250000), w, max(180, int(w * rng.uniform(0.45, 0.75))),
                    rng.choice(["speed", "type"]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs

def _fcc(nx, ny, nz, a):
    """FCC sites, four per unit cell, cell by cell (z fastest)."""
    g = np.empty((nx, ny, nz, 4, 3))
    basis = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]]) * a
    g[..., 0] = (np.arange(nx) * a)[:, None, None, None] + basis[:, 0]
    g[..., 1] = (np.arange(ny) * a)[None, :, None, None] + basis[:, 1]
    g[..., 2] = (np.arange(nz) * a)[None, None, :, None] + basis[:, 2]
    return g.reshape(-1, 3)


def _cubic(nx, ny, nz, a):
    g = np.empty((nx, ny, nz, 3))
    g[..., 0] = (np.arange(nx) * a)[:, None, None]
    g[..., 1] = (np.arange(ny) * a)[None, :, None]
    g[..., 2] = (np.arange(nz) * a)[None, None, :]
    return g.reshape(-1, 3)


def _maxwell(rng, n, sigma, zero_momentum=True):
    """Maxwell-Boltzmann velocities; zero_momentum: in opposite pairs, as the
    initializer draws them."""
    if not zero_momentum:
        return rng.standard_normal((n, 3)) * sigma
    v = np.zeros((n, 3))
    half = rng.standard_normal((n // 2, 3)) * sigma
    v[: n // 2] = half
    v[n // 2: 2 * (n // 2)] = -half
    return v


def _system(case, seed):
    """Positions, velocities, type ids, masses and box of a steps or frame case.

    Liquids: FCC sites with thermal displacements of 0.04 sigma, which keeps
    atoms apart as in a run some steps old."""
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    dims = (case["nx"], case["ny"], case["nz"])
    if case["system"] == "argon":
        a = ARGON["edge"]
        pos, box = _cubic(*dims, a), np.array(dims, dtype=np.float64) * a
        pos = np.mod(pos + rng.standard_normal(pos.shape) * 0.05, box)
        vel = _maxwell(rng, len(pos), math.sqrt(K_B * 273.15 * 0.01 / ARGON["mass"]))
        return pos, vel, np.zeros(len(pos), dtype=np.uint16), np.array([ARGON["mass"]]), box
    a = (4.0 / RHO) ** (1.0 / 3.0)
    pos, box = _fcc(*dims, a), np.array(dims, dtype=np.float64) * a
    pos = np.mod(pos + rng.standard_normal(pos.shape) * 0.04, box)
    n = len(pos)
    vel = _maxwell(rng, n, math.sqrt(T_STAR), zero_momentum=case["kind"] == "steps")
    if case.get("types", 1) == 1:
        return pos, vel, np.zeros(n, dtype=np.uint16), np.array([1.0]), box
    ids = (rng.random(n) < 0.3).astype(np.uint16)
    ids[0], ids[1] = 0, 1
    return pos, vel, ids, np.array(MIX_MASS), box


def _pairs_of(case):
    """{(type, type): (sigma, eps)} of a case."""
    if case.get("system") == "argon":
        return {(0, 0): (ARGON["sigma"], ARGON["eps"])}
    return MIX if case.get("types", 1) == 2 else {(0, 0): (1.0, 1.0)}


def _coupling(case):
    """(thermostat, T0, barostat, P0, dt) of a steps case."""
    argon = case["system"] == "argon"
    dt = 0.002 if argon else DT
    if case["coupling"] == "berendsen":
        if argon:
            return Thermostat.Berendsen(10.0), 300.0, Barostat.Berendsen(1.0, 5.0), 1.01325, dt
        return Thermostat.Berendsen(0.5), T_STAR * 100.0 / K_B, Barostat.Berendsen(1.0, 5.0), 1.0, dt
    if case["coupling"] == "nose_hoover":
        return Thermostat.NoseHoover(0.5), T_STAR * 100.0 / K_B, None, 0.0, dt
    return None, 0.0, None, 0.0, dt


def _ensemble_system(case, seed):
    """n^3 atoms per replica, n log-uniform in 4 .. 40, rho* uniform in 0.01 ..
    0.9, T* in 0.5 .. 2 (from the case); positions and velocities from the seed."""
    shape = np.random.default_rng(case["sizes_seed"])
    nrep = case["nrep"]
    ns = np.rint(np.exp(shape.uniform(np.log(4), np.log(40), nrep))).astype(int)
    rho, tst = shape.uniform(0.01, 0.9, nrep), shape.uniform(0.5, 2.0, nrep)
    p0 = rho * tst * shape.uniform(0.8, 1.2, nrep)
    rng = np.random.default_rng([seed, case["sizes_seed"]])
    pos, vel, boxes, offs = [], [], [], [0]
    for r in range(nrep):
        a = rho[r] ** (-1.0 / 3.0)
        p = _cubic(ns[r], ns[r], ns[r], a)
        box = np.full(3, ns[r] * a)
        pos.append(np.mod(p + rng.standard_normal(p.shape) * 0.02, box))
        vel.append(_maxwell(rng, len(p), math.sqrt(tst[r])))
        boxes.append(box)
        offs.append(offs[-1] + len(p))
    return np.array(offs), np.concatenate(pos), np.concatenate(vel), np.array(boxes), tst * 100.0 / K_B, p0


def _particles(case, seed):
    """The viewer's instance data of a liquid frame (12 floats a particle)."""
    rng = np.random.default_rng([seed, case["nx"], case["ny"], case["nz"]])
    a = (4.0 / RHO) ** (1.0 / 3.0)
    dims = (case["nx"], case["ny"], case["nz"])
    box = np.array(dims, dtype=np.float64) * a
    pos = _fcc(*dims, a)
    pos = np.mod(pos + rng.standard_normal(pos.shape) * 0.08, box)
    n = len(pos)
    parts = np.zeros((n, 12), dtype=np.float32)
    parts[:, 0:3] = pos
    parts[:, 3] = 1.0
    parts[:, 4:7] = rng.standard_normal((n, 3)) * math.sqrt(T_STAR)
    parts[:, 7] = 1.0
    parts[:, 8] = 1.0
    parts[:, 9] = 0.5
    parts[:, 10] = np.arange(n) % 3
    return parts, box


# ---------------------------------------------------------------------------
# the measured side

def _engine(case, **kw):
    return Engine(precision=case["precision"], reference_order=case["reference_order"],
                  skin=0.0 if case["system"] == "argon" else SKIN,
                  threads_per_atom=case["threads_per_atom"], **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "render":
        parts, box = _particles(case, seed)
        cam = rnd.framing_camera(box, case["width"], case["height"])
        mode = rnd.MODE_SPEED if case["mode"] == "speed" else rnd.MODE_TYPE
        return {"case": case, "parts": parts,
                "params": rnd.splat_params(cam, mode, speed_range=(0.0, 2.5), box=box)}
    if kind == "ensemble":
        offs, pos, vel, boxes, t0, p0 = _ensemble_system(case, seed)
        nrep = case["nrep"]
        eng = Engine(precision="mixed", skin=SKIN, persistent=True, graph_steps=50,
                     threads_per_atom=case["threads_per_atom"])
        eng.set_potential(0, 0, 1.0, 1.0)
        eng.upload_ensemble(offs, np.zeros(len(pos), dtype=np.uint16), pos, vel, [1.0], boxes)
        eng.compute_forces()
        ths = [Thermostat.Berendsen(0.5) for _ in range(nrep)]
        bas = [Barostat.Berendsen(1.0, 5.0) for _ in range(nrep)]
        eng.ensemble_set_coupling(ths, t0, bas, p0)
        eng.prepare_step(case["steps"], DT)
        return {"case": case, "engine": eng, "thermostats": ths, "barostats": bas, "out": {}}
    pos, vel, ids, mass, box = _system(case, seed)
    if kind == "frame":
        eng = _engine(case)
        for (a, b), (s, e) in _pairs_of(case).items():
            eng.set_potential(a, b, s, e)
        return {"case": case, "engine": eng, "arrays": (ids, pos, vel, mass, box), "out": {}}
    th, t0, ba, p0, dt = _coupling(case)
    st = {"case": case, "dt": dt, "th": th, "t0": t0, "ba": ba, "p0": p0, "out": {}}
    if case["api"] == "calculate":
        ParticleDatabase.add(0, "Argon", ARGON["mass"], ARGON["radius"])
        pdb = PotentialsDatabase()
        pdb.set_potential(0, 0, Potential.new_lennard_jones(ARGON["sigma"], ARGON["eps"]))
        st["pdb"], st["state"] = pdb, State(pos, vel, ids, box)
        return st
    eng = st["engine"] = _engine(case, graph_steps=case["graph_steps"])
    for (a, b), (s, e) in _pairs_of(case).items():
        eng.set_potential(a, b, s, e)
    eng.upload(ids, pos, vel, mass, box)
    eng.compute_forces()
    if case["graph_steps"]:
        eng.prepare_step(case["steps"], dt, thermostat=th, barostat=ba)
    if case["upload"]:
        st["arrays"] = (ids, pos, vel, mass, box)
    return st


def _with_coupling(out, th, ba):
    out = dict(out)
    if th is not None:
        out["lambda"], out["psi"] = th.lambda_, th.psi
    if ba is not None:
        out["myu"] = ba.myu
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        return rnd.splat(state["parts"], state["params"], case["width"], case["height"])
    eng = state.get("engine")
    if kind == "ensemble":
        eng.ensemble_step(case["steps"], DT)
        out = dict(eng.download(state["out"]))
        eng.ensemble_get_coupling()
        out["lambda"] = np.array([t.lambda_ for t in state["thermostats"]])
        out["myu"] = np.array([b.myu for b in state["barostats"]])
        return out
    if kind == "frame":
        eng.upload(*state["arrays"])
        eng.compute_forces()
        macro = [eng.macro(t) for t in range(case["types"])]
        return {"macro": macro, "state": eng.download(state["out"], fields=("force", "potential", "temp"))}
    th, ba = state["th"], state["ba"]
    if case["api"] == "calculate":
        s = state["state"]
        Integrator.VerletMethod.calculate(state["pdb"], s, state["dt"], None if ba is None else (ba, state["p0"]),
                                          None if th is None else (th, state["t0"]))
        return _with_coupling({"pos": s.positions, "vel": s.velocities, "force": s.forces,
                               "potential": s.potential, "temp": s.temp, "box": s.boundary_box}, th, ba)
    if case["upload"]:
        eng.upload(*state["arrays"])
        eng.compute_forces()
    done = 0
    while done < case["steps"]:
        n = min(case["frame_every"], case["steps"] - done)
        eng.step(n, state["dt"], thermostat=th, target_temperature=state["t0"], barostat=ba,
                 target_pressure=state["p0"])
        out = eng.download(state["out"])
        done += n
    return _with_coupling(out, th, ba)


def _atoms(case):
    n = case["nx"] * case["ny"] * case["nz"]
    return n if case.get("system") == "argon" else 4 * n


def work(case):
    """Bytes: per step the positions, velocities and forces read and written
    once (FP64), and the pass's inputs and outputs.  Operations: per step each
    interacting pair once (about 40), and about 30 an atom."""
    kind = case["kind"]
    if kind == "render":
        n, pix = _atoms(case), case["width"] * case["height"]
        return {"bytes": 48 * n + 16 * pix, "flops": 30 * n + 80 * pix}
    if kind == "ensemble":
        shape = np.random.default_rng(case["sizes_seed"])
        ns = np.rint(np.exp(shape.uniform(np.log(4), np.log(40), case["nrep"]))) ** 3
        rho = shape.uniform(0.01, 0.9, case["nrep"])
        n = float(ns.sum())
        pairs = float((ns * 2.0 / 3.0 * math.pi * 2.5 ** 3 * rho).sum())
        return {"bytes": case["steps"] * 144 * n + 88 * n, "flops": case["steps"] * (40 * pairs + 30 * n)}
    n = _atoms(case)
    per_atom = 0.035 if case["system"] == "argon" else 2.0 / 3.0 * math.pi * 2.5 ** 3 * RHO
    if kind == "frame":
        return {"bytes": n * (50 + 40), "flops": n * (40 * per_atom + 40)}
    frames = -(-case["steps"] // case["frame_every"])
    io = 88 * n * frames + (50 * n if case["upload"] else 0)
    return {"bytes": case["steps"] * 144 * n + io,
            "flops": (case["steps"] + (1 if case["upload"] else 0)) * n * (40 * per_atom + 30)}


# ---------------------------------------------------------------------------
# 64-bit torch restatement of the physics, for the error of either side

class _Exact:
    """Many independent periodic boxes at once (a single system is one box):
    LJ forces over a half pair list, velocity Verlet, Berendsen / Nose-Hoover.
    Types: an atom of type t feels only atoms of types >= t."""

    def __init__(self, pos, vel, ids, mass, boxes, offsets, pairs, skin):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = dict(dtype=torch.float64, device=dev)
        self.dev = dev
        self.x, self.v = torch.tensor(pos, **f), torch.tensor(vel, **f)
        self.ids = torch.tensor(ids.astype(np.int64), device=dev)
        self.m = torch.tensor(np.asarray(mass, dtype=np.float64)[ids], **f)
        self.box = torch.tensor(np.asarray(boxes, dtype=np.float64).reshape(-1, 3), **f)
        n = np.diff(np.asarray(offsets))
        self.nrep = len(n)
        self.rep = torch.repeat_interleave(torch.arange(self.nrep, device=dev), torch.tensor(n, device=dev))
        self.count = torch.tensor(n, **f)
        nt = max(max(p) for p in pairs) + 1
        self.nt = nt
        s, e = np.zeros((nt, nt)), np.zeros((nt, nt))
        for (a, b), (sg, ep) in pairs.items():
            s[a, b] = s[b, a] = sg
            e[a, b] = e[b, a] = ep
        self.sig, self.eps = torch.tensor(s, **f), torch.tensor(e, **f)
        self.rc = 2.5 * self.sig
        c = 0.4 ** 6                                   # (sigma / r_cut)^6
        self.ucut = 4.0 * self.eps * (c * c - c)
        self.rl = float(self.rc.max()) + skin
        self.skin = skin
        self.built = None

    def image(self, d, box):
        h = 0.5 * box
        return torch.where(d < -h, d + box, torch.where(d > h, d - box, d))

    def build(self):
        """Half pair list within rl: atoms binned into cells at least rl wide
        (boxes under three cells a side are one cell), 13 forward neighbour
        cells and the own cell."""
        nc = torch.floor(self.box / (self.rl * 1.0001)).long()
        nc[(nc < 3).any(dim=1)] = 1
        base = torch.cumsum(nc.prod(dim=1), 0)
        ncell = int(base[-1])
        base = base - nc.prod(dim=1)
        an, ab = nc[self.rep], base[self.rep]
        c = torch.minimum(torch.clamp((self.x / self.box[self.rep] * an).long(), min=0), an - 1)
        cell = ab + (c[:, 0] * an[:, 1] + c[:, 1]) * an[:, 2] + c[:, 2]
        order = torch.argsort(cell)
        cnt = torch.bincount(cell, minlength=ncell)
        start = torch.cumsum(cnt, 0) - cnt
        one = an[:, 0] == 1
        place = torch.empty_like(order)
        place[order] = torch.arange(len(order), device=self.dev)
        got_i, got_j = [], []
        rows = torch.arange(len(order), device=self.dev)
        step = 2_000_000
        for code in range(13, 27):
            o = torch.tensor([code % 3 - 1, code // 3 % 3 - 1, code // 9 - 1], device=self.dev)
            for b in range(0, len(rows), step):
                r = rows[b:b + step]
                nb = (c[r] + o) % an[r]
                cj = ab[r] + (nb[:, 0] * an[r, 1] + nb[:, 1]) * an[r, 2] + nb[:, 2]
                if code != 13:
                    r, cj = r[~one[r]], cj[~one[r]]
                k = cnt[cj]
                i = torch.repeat_interleave(r, k)
                run0 = torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
                p = torch.repeat_interleave(start[cj], k) + torch.arange(len(i), device=self.dev) - run0
                j = order[p]
                if code == 13:
                    keep = p > place[i]
                    i, j = i[keep], j[keep]
                d = self.image(self.x[j] - self.x[i], self.box[self.rep[i]])
                keep = (d * d).sum(dim=1) < self.rl * self.rl
                got_i.append(i[keep])
                got_j.append(j[keep])
        self.i, self.j = torch.cat(got_i), torch.cat(got_j)
        self.built, self.built_box = self.x.clone(), self.box.clone()

    def forces(self):
        if self.built is not None:
            d = self.x - self.built * (self.box / self.built_box)[self.rep]
            d = self.image(d, self.box[self.rep])
            moved = float((d * d).sum(dim=1).max().sqrt())
            shrink = float((self.box / self.built_box).min())
        if self.built is None or 2.0 * moved > shrink * self.rl - (self.rl - self.skin) - 1e-9:
            self.build()
        n = len(self.x)
        self.f = torch.zeros_like(self.x)
        self.u = torch.zeros(n, dtype=torch.float64, device=self.dev)
        self.w = torch.zeros_like(self.u)
        step = 50_000_000
        for b in range(0, len(self.i), step):
            i, j = self.i[b:b + step], self.j[b:b + step]
            d = self.image(self.x[j] - self.x[i], self.box[self.rep[i]])
            r2 = (d * d).sum(dim=1)
            ti, tj = self.ids[i], self.ids[j]
            keep = r2 <= self.rc[ti, tj] ** 2
            i, j, d, r2, ti, tj = i[keep], j[keep], d[keep], r2[keep], ti[keep], tj[keep]
            s2 = self.sig[ti, tj] ** 2 / r2
            s6 = s2 * s2 * s2
            e = self.eps[ti, tj]
            u = 4.0 * e * (s6 * s6 - s6) - self.ucut[ti, tj]
            w = 24.0 * e * (s6 - 2.0 * s6 * s6)        # r dU/dr = F . r
            g = d * (w / r2)[:, None]
            if self.nt == 1:
                self.f.index_add_(0, i, g)
                self.f.index_add_(0, j, -g)
                for a, q in ((self.u, u), (self.w, w)):
                    a.index_add_(0, i, q)
                    a.index_add_(0, j, q)
            else:
                for a, q, fi, fj in ((i, g, ti, tj), (j, -g, tj, ti)):
                    see = fj >= fi
                    self.f.index_add_(0, a[see], q[see])
                    self.u.index_add_(0, a[see], u[see])
                    self.w.index_add_(0, a[see], w[see])

    def per_box(self, q):
        out = torch.zeros((self.nrep,) + q.shape[1:], dtype=torch.float64, device=self.dev)
        return out.index_add_(0, self.rep, q)

    def thermal(self):
        vcm = self.per_box(self.v) / self.count[:, None]
        d = self.v - vcm[self.rep]
        return self.per_box(0.5 * self.m * (d * d).sum(dim=1))

    def temperature(self):
        return 2.0 * self.thermal() / (3.0 * self.count * K_B) * 100.0

    def step(self, dt, th=None, t0=None, ba=None, p0=None):
        """th: ["berendsen", tau, lambda] or ["nose_hoover", tau, lambda, psi];
        ba: [beta, tau, mu]."""
        if ba is not None:
            p = (2.0 * self.thermal() - 0.5 * self.per_box(self.w)) / self.box.prod(dim=1) / 3.0
            m3 = 1.0 + dt * ba[0] / ba[1] * (p - p0)
            ba[2] = torch.sign(m3) * m3.abs() ** (1.0 / 3.0)
        if th is not None:
            t = self.temperature()
            if th[0] == "berendsen":
                th[2] = torch.sqrt(1.0 + dt / th[1] * (t0 / t - 1.0))
            else:
                th[3] = th[3] - (t0 / t - 1.0) / th[1] * (dt / 2.0)
                th[2] = torch.exp(-th[3] * dt / 2.0)
        kick = (dt / (2.0 * self.m))[:, None]
        self.v = self.v + self.f * kick
        if th is not None:
            if th[0] == "nose_hoover":
                th[3] = th[3] - (t0 / self.temperature() - 1.0) / th[1] * (dt / 2.0)
            self.v = self.v * th[2][self.rep][:, None]
        self.x = self.x + self.v * dt
        box = self.box[self.rep]
        self.x = torch.where(self.x < 0.0, self.x + box, torch.where(self.x >= box, self.x - box, self.x))
        self.forces()
        self.v = self.v + self.f * kick
        if ba is not None:
            self.box = self.box * ba[2][:, None]
            self.x = self.x * ba[2][self.rep][:, None]

    def state(self):
        return {"pos": self.x, "vel": self.v, "force": self.f, "potential": self.u, "temp": self.w}


def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        return None   # which sphere a pixel shows flips with the last bit of a silhouette
    if kind == "ensemble":
        offs, pos, vel, boxes, t0, p0 = _ensemble_system(case, seed)
        e = _Exact(pos, vel, np.zeros(len(pos), dtype=np.uint16), [1.0], boxes, offs, {(0, 0): (1.0, 1.0)}, 0.4)
        e.forces()
        t0, p0 = (torch.tensor(q, dtype=torch.float64, device=e.dev) for q in (t0, p0))
        th, ba = ["berendsen", 0.5, None], [1.0, 5.0, None]
        for _ in range(case["steps"]):
            e.step(DT, th, t0, ba, p0)
        return dict(e.state(), box=e.box, **{"lambda": th[2], "myu": ba[2]})
    pos, vel, ids, mass, box = _system(case, seed)
    skin = 0.1 if case["system"] == "argon" else 0.4
    e = _Exact(pos, vel, ids, mass, box, [0, len(pos)], _pairs_of(case), skin)
    e.forces()
    if kind == "frame":
        macro = []
        for t in range(case["types"]):
            of = e.ids == t
            v, m = e.v[of], float(mass[t])
            n = len(v)
            vcm = v.mean(dim=0)
            d2 = ((v - vcm) ** 2).sum()
            th = float(0.5 * m * d2)
            macro.append({"kinetic_energy": float(0.5 * m * (v * v).sum()), "potential_energy": float(e.u[of].sum() / 2),
                          "thermal_energy": th, "temperature": 2.0 * th / (3.0 * n * K_B) * 100.0,
                          "pressure": float((m * d2 - 0.5 * e.w[of].sum()) / e.box[0].prod() / 3.0),
                          "com_velocity": vcm, "momentum": v.sum(dim=0) * m, "count": n})
        s = e.state()
        return {"macro": macro, "state": dict({k: s[k] for k in ("force", "potential", "temp")}, box=e.box[0])}
    th, t0, ba, p0, dt = _coupling(case)
    if case["api"] == "calculate":
        e.f, e.u, e.w = (torch.zeros_like(q) for q in (e.f, e.u, e.w))   # a fresh State carries no forces
    one = torch.zeros(1, dtype=torch.float64, device=e.dev)
    xt = None if th is None else [th.kind, th.tau, one, one]
    xb = None if ba is None else [ba.beta, ba.tau, one]
    for _ in range(case["steps"]):
        e.step(dt, xt, t0, xb, p0)
    out = dict(e.state(), box=e.box[0])
    if xt is not None:
        out["lambda"], out["psi"] = float(xt[2]), float(xt[3])
    if xb is not None:
        out["myu"] = float(xb[2])
    return out
