"""Performance cases of the GB300 LULESH Lagrange-leapfrog step.

Each case is one way a program uses the framework: the resident time loop
(host TimeIncrement or CUDA graph), single steps, the drop-in call on host
buffers, an ensemble in a batch pool, the serving loop. Sizes are the
repository's own (s = 8 of the smoke run to the benchmark's s = 150, r in
{11, 16, 21}) and odd ones between them.

Single-problem cases start from a blast in mid-run, which is what most cycles
of a run see: a compressed shell behind a shock at a seeded radius, material
moving and under pressure inside it, material at rest outside. A state that
has run `horizon` cycles starts over from its first one.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "lulesh-task-based-hpx_gb300"

NODE = ("x", "y", "z", "xd", "yd", "zd", "xdd", "ydd", "zdd", "fx", "fy", "fz")
ELEM = ("e", "p", "q", "ql", "qq", "v", "vnew", "delv", "vdov", "arealg", "ss")
TIMES = ("time", "deltatime", "dtcourant", "dthydro")
STATE = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")  # what a cycle reads of the last one's results


def package():
    if "lulesh_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("lulesh_gb300", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["lulesh_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["lulesh_gb300"]


def listed():
    return [
        # one cycle on a small mesh, the host holding the time loop: latency and launches
        {"name": "step_s8_fp64", "kind": "step", "s": 8, "r": 11, "precision": "fp64", "cycles": 1},
        # the reference's default problem (--s 30 --r 11) in the host time loop
        {"name": "loop_s30_fp64", "kind": "loop", "s": 30, "r": 11, "precision": "fp64", "cycles": 20},
        # the smallest size of the reference's published sweep, replayed from the CUDA graph
        {"name": "graph_s45_fp64", "kind": "graph", "s": 45, "r": 11, "precision": "fp64", "cycles": 32},
        # an odd size in the middle of the sweep
        {"name": "loop_s91_fp64", "kind": "loop", "s": 91, "r": 16, "precision": "fp64", "cycles": 10},
        # the headline problem: s=150 r=21 in the host time loop
        {"name": "loop_s150_fp64", "kind": "loop", "s": 150, "r": 21, "precision": "fp64", "cycles": 10},
        # the drop-in call of a program that keeps its Domain in (pinned) host memory
        {"name": "dropin_s45_fp64", "kind": "dropin", "s": 45, "r": 11, "precision": "fp64", "cycles": 1},
        {"name": "dropin_s150_fp64", "kind": "dropin", "s": 150, "r": 21, "precision": "fp64", "cycles": 1},
        # the bit-exact variant, as a reference run for validation
        {"name": "loop_s60_exact", "kind": "loop", "s": 60, "r": 11, "precision": "fp64_exact", "cycles": 10},
        # mixed precision at an odd size (host loop) and at s=120 (graph)
        {"name": "loop_s37_mixed", "kind": "loop", "s": 37, "r": 16, "precision": "mixed", "cycles": 20},
        {"name": "graph_s120_mixed", "kind": "graph", "s": 120, "r": 21, "precision": "mixed", "cycles": 20},
        # an ensemble of uneven problems in one pool (parameter study)
        {"name": "ensemble_fp64", "kind": "ensemble", "n": 14, "smin": 16, "smax": 64, "precision": "fp64",
         "cycles": 8},
        # the serving loop: a burst of requests, admitted, run and reported
        {"name": "serve_mixed", "kind": "serve", "n": 16, "smin": 20, "smax": 90, "precision": "mixed",
         "cycles": 48},
    ]


# What one zone-cycle costs in units of a double zone-cycle; the cycles of a
# pass are cut so that a drawn case stays below the largest listed one.
COST = {"fp64": 1.0, "fp64_exact": 3.0, "mixed": 0.4}


def draw(rng):
    kind = rng.choice(("step", "loop", "loop", "graph", "graph", "dropin", "ensemble", "serve"))
    precision = rng.choice(("fp64", "fp64", "fp64", "mixed", "mixed", "fp64_exact"))
    if kind in ("ensemble", "serve"):
        precision = "mixed" if precision == "fp64_exact" else precision
        smin = rng.randint(16, 24)
        smax = rng.randint(smin + 8, 56)
        return {"kind": kind, "n": rng.randint(6, 14), "smin": smin, "smax": smax, "precision": precision,
                "cycles": rng.randint(4, 10) if kind == "ensemble" else rng.randint(20, 48)}
    s = int(round(math.exp(rng.uniform(math.log(8), math.log(140)))))
    cycles = 1
    if kind in ("loop", "graph"):
        cycles = rng.randint(8, 32)
        cycles = max(1, min(cycles, int(8 * 150 ** 3 / (COST[precision] * s ** 3))))
    return {"kind": kind, "s": s, "r": rng.choice((11, 16, 21)), "precision": precision, "cycles": cycles}


# --- inputs -------------------------------------------------------------------


def blast(s, seed, device):
    """A blast in mid-run on the s^3 mesh: the STATE arrays (node arrays
    (s+1)^3, element arrays s^3, in z, y, x order) and the first time step."""
    rng = np.random.default_rng(seed)
    radius = 1.125 * rng.uniform(0.6, 1.0)   # of the shock
    stretch = rng.uniform(0.2, 0.3)          # the interior is spread out, the shell behind the shock dense
    speed = 100.0 * rng.lognormal(0.0, 0.25)
    waves = [(rng.uniform(2.0, 6.0, 3), rng.uniform(0.0, 2 * math.pi), rng.uniform(0.01, 0.03)) for _ in range(3)]
    line = torch.arange(s + 1, dtype=torch.float64, device=device) * 1.125 / s
    z, y, x = torch.meshgrid(line, line, line, indexing="ij")
    r = torch.sqrt(x * x + y * y + z * z) / radius
    inside = (r < 1.0).double()
    ripple = torch.zeros_like(x)
    for k, phase, amp in waves:
        ripple += amp * torch.cos(k[0] * x + k[1] * y + k[2] * z + phase)
    grow = 1.0 + inside * stretch * (1.0 - r * r) * (1.0 + ripple)
    fast = inside * speed / radius * (1.0 + ripple)
    st = {"x": x * grow, "y": y * grow, "z": z * grow, "xd": x * fast, "yd": y * fast, "zd": z * fast}
    h = 1.125 / s
    v = hex_volume(*(corners(st[f]) for f in "xyz")) / (h * h * h)
    rm = sum(corners(r)) / 8
    moving = (rm < 1.0).double()
    v = torch.where(moving > 0, v, torch.ones_like(v))
    st["v"] = v
    st["e"] = moving * speed * speed * (0.4 + 0.6 * rm * rm) * (1.0 + sum(corners(ripple)) / 8)
    st["p"] = 2.0 / 3.0 * st["e"] / v
    st["q"] = moving * torch.clamp(rm - 0.9, min=0.0) * 2.0 * st["p"]
    st["ss"] = torch.sqrt(10.0 / 9.0 * st["e"])
    return {f: a.contiguous() for f, a in st.items()}, 0.05 * h / speed


def specs(case, seed):
    """Problems of an ensemble or a burst of requests: sizes over the range, seeded energies."""
    rng = np.random.default_rng(seed)
    n, lo, hi = case["n"], case["smin"], case["smax"]
    out = []
    for k in range(n):
        s = int(round(lo * (hi / lo) ** (k / (n - 1))))
        out.append({"s": s, "nr": (11, 16, 21)[k % 3], "energy_scale": float(rng.lognormal(0.0, 0.25))})
    return out


class Field:
    """A host Domain's array that keeps its Domain alive."""

    def __init__(self, dom, name):
        self.dom = dom
        self.__array_interface__ = getattr(dom, name).__array_interface__


class Single:
    """A handle, its host Domain (pinned, as a program that downloads results keeps it) and the first state."""

    def __init__(self, case, seed):
        lul = package()
        st, dt = blast(case["s"], seed, "cuda")
        self.first = {f: a.reshape(-1).cpu().numpy() for f, a in st.items()}
        self.dt = dt
        self.horizon = 400
        self.dom = lul.HostDomain(case["s"], case["r"])
        self.dom.pin()
        self.fields = {f: np.asarray(Field(self.dom, f)) for f in NODE + ELEM}
        self.load()
        self.dev = lul.Device(self.dom, case["precision"])

    def load(self):
        for f in NODE[6:] + ("ql", "qq", "vnew", "delv", "vdov", "arealg"):
            getattr(self.dom, f)[:] = 0.0
        for f, a in self.first.items():
            getattr(self.dom, f)[:] = a
        ts = self.dom.time_state
        ts.time, ts.cycle, ts.deltatime, ts.stoptime = 0.0, 0, self.dt, 1.0
        ts.dtcourant = ts.dthydro = 1.0e20

    def out(self):
        ts = self.dom.time_state
        r = dict(self.fields)
        r.update({f: getattr(ts, f) for f in TIMES})
        r["cycle"] = int(ts.cycle)
        return r


class Ensemble:
    """A batch pool with its problems, and a host Domain of each for its fields."""

    def __init__(self, case, seed):
        lul = package()
        self.specs = specs(case, seed)
        need = sum(lul.Batch.footprint(case["precision"], p["s"]) for p in self.specs)
        self.batch = lul.Batch(case["precision"], pool_bytes=int(need * 1.05) + (16 << 20), max_slots=len(self.specs))
        self.slots = [self.batch.admit(**p) for p in self.specs]
        self.doms = [lul.HostDomain(p["s"], p["nr"], energy_scale=p["energy_scale"]) for p in self.specs]
        self.fields = {"%s_%d" % (f, k): np.asarray(Field(dom, f)) for k, dom in enumerate(self.doms) for f in "epqv"}
        self.active = {slot: True for slot in self.slots}


def prepare(case, seed):
    package().set_device(0)
    if case["kind"] == "ensemble":
        return case, Ensemble(case, seed)
    if case["kind"] == "serve":
        reqs = [dict(p, arrival_s=0.0, max_cycles=case["cycles"] + 2 * (k % 5))
                for k, p in enumerate(specs(case, seed))]
        return case, reqs
    return case, Single(case, seed)


def run(state):
    case, st = state
    lul = package()
    if case["kind"] == "serve":
        results, _ = lul.serve(st, case["precision"], hbm_budget=4 << 30, max_slots=64, sync_ms=20.0)
        return {"e0": np.array([r["e0"] for r in results]), "cycles": np.array([r["cycles"] for r in results]),
                "zone_cycles": np.array([r["zone_cycles"] for r in results])}
    if case["kind"] == "ensemble":
        for k, (slot, p) in enumerate(zip(st.slots, st.specs)):  # a finished problem makes room for the next one
            if not st.active[slot]:
                st.batch.retire(slot)
                st.slots[k] = st.batch.admit(**p)
        st.batch.run(case["cycles"])
        status = {x["slot"]: x for x in st.batch.status()}
        st.active = {slot: bool(status[slot]["active"]) for slot in st.slots}
        for dom, slot in zip(st.doms, st.slots):
            code = lul.library().lulesh_batch_download(st.batch._h, slot, dom.view_ptr, lul.F_EPQ | lul.F_V)
            if code != lul.OK:
                raise lul.LuleshError(code, "lulesh_batch_download")
        r = dict(st.fields)
        for f in TIMES + ("cycle",):
            r[f] = np.array([status[slot][f] for slot in st.slots])
        return r
    ts = st.dom.time_state
    if ts.cycle >= st.horizon:
        st.load()
        st.dev.upload()
    if case["kind"] == "dropin":
        st.dom.time_increment()
        st.dev.leapfrog()
        return st.out()
    if case["kind"] == "step":
        st.dom.time_increment()
        ts.dtcourant, ts.dthydro = st.dev.step(ts.deltatime)
    elif case["kind"] == "graph":
        st.dev.run_graph(ts.cycle + case["cycles"], case["cycles"])
    else:
        st.dev.run(ts.cycle + case["cycles"])
    st.dev.download()
    return st.out()


def work(case):
    """Per zone-cycle: the mutable state read (11 doubles), the constants
    (nodal mass, reference volume and mass, node list, corner list, face
    neighbours, boundary mask, order and repeat count), every result written
    (23 doubles), and the reference's 3,300 floating-point operations; the
    results go to the host once a pass (the drop-in's inputs come from there)."""
    if case["kind"] in ("ensemble", "serve"):
        zones = sum(p["s"] ** 3 for p in specs(case, 0))
    else:
        zones = case["s"] ** 3
    zc = zones * case["cycles"]
    down = {"serve": 0, "ensemble": 4 * 8 * zones}.get(case["kind"], 23 * 8 * zones)
    return {"bytes": zc * (11 * 8 + 3 * 8 + 104 + 23 * 8) + down, "flops": zc * 3300}


# --- the cycle in plain 64-bit torch ------------------------------------------


def corners(a):
    """The 8 corner values of each element, in the node list's order."""
    n = [a[dz:a.shape[0] - 1 + dz, dy:a.shape[1] - 1 + dy, dx:a.shape[2] - 1 + dx]
         for dz, dy, dx in ((0, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0), (1, 0, 0), (1, 0, 1), (1, 1, 1), (1, 1, 0))]
    return n


def to_nodes(f, s):
    """Corner values summed into their nodes."""
    out = torch.zeros((s + 1, s + 1, s + 1), dtype=torch.float64, device=f[0].device)
    for k, (dz, dy, dx) in enumerate(((0, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0), (1, 0, 0), (1, 0, 1), (1, 1, 1),
                                      (1, 1, 0))):
        out[dz:dz + s, dy:dy + s, dx:dx + s] += f[k]
    return out


def cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


FACES = ((0, 1, 2, 3), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0), (4, 7, 6, 5))
GAMMA = ((1, 1, -1, -1, -1, -1, 1, 1), (1, -1, -1, 1, -1, 1, 1, -1), (1, -1, 1, -1, 1, -1, 1, -1),
         (-1, 1, -1, 1, 1, -1, 1, -1))
# corners of the volume derivative's six products, for each corner
DERIV = ((0, 1, 2, 3, 4, 5, 7), (3, 0, 1, 2, 7, 4, 6), (2, 3, 0, 1, 6, 7, 5), (1, 2, 3, 0, 5, 6, 4),
         (4, 7, 6, 5, 0, 3, 1), (5, 4, 7, 6, 1, 0, 2), (6, 5, 4, 7, 2, 1, 3), (7, 6, 5, 4, 3, 2, 0))


def diff(p, i, j):
    return tuple(c[i] - c[j] for c in p)


def add(a, b):
    return tuple(u + w for u, w in zip(a, b))


def hex_volume(x, y, z):
    p = (x, y, z)
    d = lambda i, j: diff(p, i, j)  # noqa: E731
    return (dot(add(d(3, 1), d(7, 2)), cross(d(6, 3), d(2, 0))) + dot(add(d(4, 3), d(5, 7)), cross(d(6, 4), d(7, 0))) +
            dot(add(d(1, 4), d(2, 5)), cross(d(6, 1), d(5, 0)))) / 12.0


def directions(v):
    """Sums of the four body diagonals of v along xi, eta, zeta: 8 x its centre gradient."""
    d60, d53, d71, d42 = v[6] - v[0], v[5] - v[3], v[7] - v[1], v[4] - v[2]
    return (d60 + d53 - d71 - d42, d60 - d53 + d71 - d42, d60 + d53 + d71 + d42)


def cofactor(J):
    """c[a][d] of J[a][d] (a the coordinate, d the direction)."""
    col = [[J[a][d] for a in range(3)] for d in range(3)]
    c = [cross(col[(d + 1) % 3], col[(d + 2) % 3]) for d in range(3)]
    return [[c[d][a] for d in range(3)] for a in range(3)]


def limiter(dv, axis):
    """Monotonic limiter along one axis: symmetry on the minus face, free surface on the plus face."""
    norm = 1.0 / (dv + 1.0e-36)
    zero = torch.zeros_like(dv.narrow(axis, 0, 1))
    m = torch.cat((dv.narrow(axis, 0, 1), dv.narrow(axis, 0, dv.shape[axis] - 1)), axis) * norm
    p = torch.cat((dv.narrow(axis, 1, dv.shape[axis] - 1), zero), axis) * norm
    phi = 0.5 * (m + p)
    phi = torch.minimum(phi, torch.minimum(2.0 * m, 2.0 * p))
    return torch.clamp(phi, 0.0, 1.0)


def cut(a, c):
    return torch.where(a.abs() < c, torch.zeros_like(a), a)


def eos(e0, p0, q0, ql, qq, v, delv):
    def pressure(b, e):
        return torch.clamp(cut(b * e, 1.0e-7), min=0.0)

    def sound(e, w, p):
        return torch.sqrt(torch.clamp(2.0 / 3.0 * (e + w * p), min=1.111111e-37))

    zero = torch.zeros_like(e0)
    opening = delv > 0.0
    vh = v - 0.5 * delv
    e = e0 - 0.5 * delv * (p0 + q0)
    ph = pressure(2.0 / 3.0 / vh, e)
    q = torch.where(opening, zero, sound(e, vh, ph) * ql + qq)
    e = cut(e + 0.5 * delv * (3.0 * (p0 + q0) - 4.0 * (ph + q)), 1.0e-7)
    p = pressure(2.0 / 3.0 / v, e)
    qt = torch.where(opening, zero, sound(e, v, p) * ql + qq)
    e = cut(e - (7.0 * (p0 + q0) - 8.0 * (ph + q) + (p + qt)) * delv / 6.0, 1.0e-7)
    p = pressure(2.0 / 3.0 / v, e)
    q = torch.where(opening, q, cut(sound(e, v, p) * ql + qq, 1.0e-7))
    return e, p, q, sound(e, v, p)


def next_dt(t):
    """The reference's TimeIncrement (no fixed step)."""
    target = t["stoptime"] - t["time"]
    if t["cycle"] != 0:
        new = 1.0e20
        if t["dtcourant"] < new:
            new = t["dtcourant"] / 2.0
        if t["dthydro"] < new:
            new = t["dthydro"] * 2.0 / 3.0
        ratio = new / t["deltatime"]
        if 1.0 <= ratio < 1.1:
            new = t["deltatime"]
        elif ratio > 1.2:
            new = t["deltatime"] * 1.2
        t["deltatime"] = min(new, 1.0e-2)
    if t["deltatime"] < target < 4.0 * t["deltatime"] / 3.0:
        target = 2.0 * t["deltatime"] / 3.0
    t["deltatime"] = min(target, t["deltatime"])
    t["time"] += t["deltatime"]
    t["cycle"] += 1


def cycle(f, const, t, s):
    """One Lagrange-leapfrog cycle of the Sedov cube on the fields f."""
    next_dt(t)
    dt = t["deltatime"]
    mass, volo, emass = const
    # corner forces: stress (p + q on each face's area vector) and hourglass
    p = tuple(corners(f[a]) for a in "xyz")
    force = [[0.0] * 8 for _ in range(3)]
    press = f["p"] + f["q"]
    for a, b, c, d in FACES:
        area = cross(diff(p, d, b), diff(p, c, a))
        for k in (a, b, c, d):
            for ax in range(3):
                force[ax][k] = force[ax][k] + 0.125 * press * area[ax]
    det = volo * f["v"]
    grad = [[None] * 8 for _ in range(3)]
    for k, p0, p1, p2, p3, p4, p5 in DERIV:
        for ax in range(3):
            u, w = p[(ax + 1) % 3], p[(ax + 2) % 3]
            grad[ax][k] = ((u[p1] + u[p2]) * (w[p0] + w[p1]) - (u[p0] + u[p1]) * (w[p1] + w[p2]) +
                           (u[p0] + u[p4]) * (w[p3] + w[p4]) - (u[p3] + u[p4]) * (w[p0] + w[p4]) -
                           (u[p2] + u[p5]) * (w[p3] + w[p5]) + (u[p3] + u[p5]) * (w[p2] + w[p5])) / 12.0
    vel = tuple(corners(f[a]) for a in ("xd", "yd", "zd"))
    coef = -0.03 * f["ss"] * emass * det.pow(-1.0 / 3.0)
    for g in GAMMA:
        mode = [sum(g[k] * p[ax][k] for k in range(8)) / det for ax in range(3)]
        shape = [g[k] - sum(grad[ax][k] * mode[ax] for ax in range(3)) for k in range(8)]
        for ax in range(3):
            h = coef * sum(shape[k] * vel[ax][k] for k in range(8))
            for k in range(8):
                force[ax][k] = force[ax][k] + shape[k] * h
    del grad, shape
    # nodes
    for ax, a in enumerate("xyz"):
        f["f" + a] = to_nodes(force[ax], s)
        acc = f["f" + a] / mass
        acc.narrow(2 - ax, 0, 1).zero_()
        f[a + "dd"] = acc
        f[a + "d"] = cut(f[a + "d"] + acc * dt, 1.0e-7)
        f[a] = f[a] + f[a + "d"] * dt
    del force
    # kinematics
    p = tuple(corners(f[a]) for a in "xyz")
    volume = hex_volume(*p)
    f["vnew"] = volume / volo
    f["delv"] = f["vnew"] - f["v"]
    face = None
    for a, b, c, d in FACES:
        n = cross(diff(p, d, b), diff(p, c, a))
        face = dot(n, n) if face is None else torch.maximum(face, dot(n, n))
    f["arealg"] = 2.0 * volume / torch.sqrt(face)
    X = [directions(c) for c in p]
    V = [directions(corners(f[a])) for a in ("xd", "yd", "zd")]
    c = cofactor(X)
    vol = volo * f["vnew"]
    dv, dx = [], []
    for d in range(3):
        n2 = sum(c[a][d] ** 2 for a in range(3))
        dx.append(16.0 * vol / torch.sqrt(n2 + 2.56e-34))
        dv.append(sum(c[a][d] * V[a][d] for a in range(3)) / (64.0 * (vol + 1.0e-36)))
    J = [[X[a][d] - 0.5 * dt * V[a][d] for d in range(3)] for a in range(3)]
    c = cofactor(J)
    f["vdov"] = sum(c[a][d] * V[a][d] for a in range(3) for d in range(3)) / sum(c[0][d] * J[0][d] for d in range(3))
    f["v"] = torch.where((f["vnew"] - 1.0).abs() < 1.0e-10, torch.ones_like(volo), f["vnew"])
    # q terms
    ql, qq = torch.zeros_like(volo), torch.zeros_like(volo)
    for d in range(3):
        phi = limiter(dv[d], 2 - d)
        push = torch.clamp(dv[d] * dx[d], max=0.0)
        ql += push * (1.0 - phi)
        qq += push * push * (1.0 - phi * phi)
    rho = emass / vol
    still = f["vdov"] > 0.0
    f["ql"] = torch.where(still, torch.zeros_like(ql), -0.5 * rho * ql)
    f["qq"] = torch.where(still, torch.zeros_like(qq), 2.0 / 3.0 * rho * qq)
    f["e"], f["p"], f["q"], f["ss"] = eos(f["e"], f["p"], f["q"], f["ql"], f["qq"], f["vnew"], f["delv"])
    # time constraints
    dtf = f["ss"] ** 2 + torch.where(f["vdov"] < 0.0, 256.0 * f["arealg"] ** 2 * f["vdov"] ** 2, torch.zeros_like(volo))
    moves = f["vdov"] != 0.0
    big = torch.full_like(volo, 1.0e20)
    t["dtcourant"] = float(torch.where(moves, f["arealg"] / torch.sqrt(dtf), big).min())
    t["dthydro"] = float(torch.where(moves, 0.1 / (f["vdov"].abs() + 1.0e-20), big).min())


def constants(s, device):
    line = torch.arange(s + 1, dtype=torch.float64, device=device) * 1.125 / s
    z, y, x = torch.meshgrid(line, line, line, indexing="ij")
    volo = hex_volume(corners(x), corners(y), corners(z))
    return to_nodes([volo / 8.0] * 8, s), volo, volo


def sedov(p, device):
    """The initial state of a problem: energy in the origin element, all at rest."""
    s = p["s"]
    line = torch.arange(s + 1, dtype=torch.float64, device=device) * 1.125 / s
    z, y, x = torch.meshgrid(line, line, line, indexing="ij")
    f = {"x": x, "y": y, "z": z}
    for a in ("xd", "yd", "zd"):
        f[a] = torch.zeros_like(x)
    volo = constants(s, device)[1]
    for a in ("e", "p", "q", "ss"):
        f[a] = torch.zeros_like(volo)
    f["v"] = torch.ones_like(volo)
    e0 = 3.948746e7 * (s / 45.0) ** 3 * p["energy_scale"]
    f["e"][0, 0, 0] = e0
    return f, 0.5 * float(volo[0, 0, 0]) ** (1.0 / 3.0) / math.sqrt(2.0 * e0), 1.0e-2


def solve(f, dt, stoptime, cycles, s, device):
    t = {"time": 0.0, "cycle": 0, "deltatime": dt, "stoptime": stoptime, "dtcourant": 1.0e20, "dthydro": 1.0e20}
    const = constants(s, device)
    while t["cycle"] < cycles and t["time"] < t["stoptime"]:
        cycle(f, const, t, s)
    return t


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "serve":
        e0, cycles = [], []
        problems = specs(case, seed)
        for k, p in enumerate(problems):
            f, dt, stop = sedov(p, device)
            cycles.append(solve(f, dt, stop, case["cycles"] + 2 * (k % 5), p["s"], device)["cycle"])
            e0.append(float(f["e"][0, 0, 0]))
        return {"e0": np.array(e0), "cycles": np.array(cycles),
                "zone_cycles": np.array([c * p["s"] ** 3 for c, p in zip(cycles, problems)])}
    if case["kind"] == "ensemble":
        r, ts = {}, []
        for k, p in enumerate(specs(case, seed)):
            f, dt, stop = sedov(p, device)
            ts.append(solve(f, dt, stop, case["cycles"], p["s"], device))
            r.update({"%s_%d" % (a, k): f[a].reshape(-1) for a in ("e", "p", "q", "v")})
        r.update({a: np.array([t[a] for t in ts]) for a in TIMES + ("cycle",)})
        return r
    f, dt = blast(case["s"], seed, device)
    t = solve(f, dt, 1.0, case["cycles"], case["s"], device)
    r = {a: f[a].reshape(-1) for a in NODE + ELEM}
    r.update({a: t[a] for a in TIMES})
    r["cycle"] = t["cycle"]
    return r
