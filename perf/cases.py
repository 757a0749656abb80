"""The library's work as its users run it: cases, inputs and one pass of each.

Five kinds of call, each through the public entry points (the Python classes
over the C ABI, and ``dpg_load_state`` of include/dpg.h where a program loads a
new configuration into a handle that it keeps):

forces  a configuration is loaded, its neighbour lists are set up, and its
        forces, energies, pressure and contacts are read: what an analysis of
        stored states does, and how every run begins;
nve     a configuration is loaded and integrated: plain, damped or with walls;
fire    a configuration is loaded and relaxed by a bounded number of FIRE
        iterations (targets that do not fire);
bumpy   the same two for rigid bumpy bodies;
ens     a batch of independent systems goes in from the host, is minimised by
        FIRE towards max|F| <= 1e-13, and comes back to the host.

Starts are uniform-random positions at the packing fractions of the repository's
workloads (0.80 to 0.86), bidisperse radii 0.5 / 0.7 or polydisperse
U[0.4, 0.6], velocities Gaussian.  FP64 is the drop-in arithmetic, mixed the
FP32 pair forces.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "dpcuda-v2_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import dpcuda_gb300 as dpg  # noqa: E402
from dpcuda_gb300.disk import DEVICE, DP, check  # noqa: E402
from dpcuda_gb300.init import bumpy_vertex_radius  # noqa: E402

C = dpg.lib.C
BI = ("cell", 1.7 / 1.4, 0.2, 8.0, 0.5)         # d_max + 0.3: the bidisperse workloads
POLY = ("cell", 1.5 / 1.2, 0.1732, 8.0, 0.5)    # the 2^20 workload
BUMPY = ("cell", 1.5, 0.2, 8.0, 0.5)


def listed():
    return [
        # one small stored state analysed: latency of the setup path
        dict(name="forces-n256-fp64", kind="forces", n=256, radii="bi", phi=0.84, precision="fp64"),
        # a large stored state, a size that is no power of two
        dict(name="forces-n131071-fp64", kind="forces", n=131071, radii="bi", phi=0.84, precision="fp64"),
        # the smallest systems of the jamming workload, here in a plain NVE run
        dict(name="nve-n64-fp64", kind="nve", n=64, radii="bi", phi=0.80, precision="fp64", steps=500,
             dt=1e-2, temp=1e-4, option="plain"),
        # the plain NVE workload: 1024 disks at phi 0.80, T 1e-4, dt 1e-2
        dict(name="nve-n1024-fp64", kind="nve", n=1024, radii="bi", phi=0.80, precision="fp64", steps=1000,
             dt=1e-2, temp=1e-4, option="plain"),
        # mixed precision with damping, at a ragged size
        dict(name="damped-n10007-mixed", kind="nve", n=10007, radii="bi", phi=0.80, precision="mixed", steps=300,
             dt=1e-2, temp=1e-4, option="damped"),
        # the large-N throughput workload in both precisions
        dict(name="nve-n1048576-fp64", kind="nve", n=1048576, radii="poly", phi=0.84, precision="fp64", steps=20,
             dt=1e-2, temp=1e-3, option="plain"),
        dict(name="nve-n1048576-mixed", kind="nve", n=1048576, radii="poly", phi=0.84, precision="mixed", steps=40,
             dt=1e-2, temp=1e-3, option="plain"),
        # the drop-in FIRE minimisation of the headline configuration
        dict(name="fire-n16384-fp64", kind="fire", n=16384, radii="bi", phi=0.86, precision="fp64", steps=400),
        # the rigid-body workload: 4096 bodies of 20 / 28 vertices
        dict(name="bumpy-nve-n4096-fp64", kind="bumpy", n=4096, phi=0.80, precision="fp64", steps=100, dt=5e-3,
             temp=1e-4, method="nve"),
        # a small, odd number of rigid bodies relaxed in mixed precision
        dict(name="bumpy-fire-n301-mixed", kind="bumpy", n=301, phi=0.80, precision="mixed", steps=100, dt=5e-3,
             temp=0.0, method="fire"),
        # the headline batch: 16 systems of 16384 disks (their first iterations)
        dict(name="ens-16x16384-mixed", kind="ens", systems=16, n_lo=16384, n_hi=16384, pick=1, phi=0.86,
             precision="mixed", steps=300),
        # an uneven batch of the jamming ensemble's sizes, through all phases:
        # its small systems converge, its large ones run to the cap
        dict(name="ens-24-uneven-mixed", kind="ens", systems=24, n_lo=64, n_hi=4096, pick=2, phi=0.86,
             precision="mixed", steps=10000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forces", "nve", "nve", "nve", "fire", "fire", "bumpy", "bumpy", "ens", "ens"])
    prec = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "ens":
        lo, hi = sorted((_log(rng, 64, 16384), _log(rng, 64, 16384)))
        s = _log(rng, 1, 24)
        return dict(kind=kind, systems=s, n_lo=lo, n_hi=hi, pick=rng.randrange(1000), phi=rng.uniform(0.80, 0.90),
                    precision="mixed", steps=max(100, min(3000, 5_000_000 // (s * hi))))
    if kind == "bumpy":
        n = _log(rng, 32, 4096)
        return dict(kind=kind, n=n, phi=rng.uniform(0.60, 0.82), precision=prec, steps=rng.randint(40, 100), dt=5e-3,
                    temp=10 ** rng.uniform(-4, -2), method=rng.choice(["nve", "fire"]))
    if kind == "fire":
        n = _log(rng, 64, 65536)
        return dict(kind=kind, n=n, radii="bi", phi=rng.uniform(0.80, 0.90), precision=prec,
                    steps=max(60, min(400 if prec == "fp64" else 200, 6_000_000 // n)))
    n = _log(rng, 64, 1048576)
    radii = "poly" if n > 100000 else rng.choice(["bi", "poly"])
    c = dict(kind=kind, n=n, radii=radii, phi=rng.uniform(0.70, 0.86), precision=prec)
    if kind == "nve":
        c.update(steps=max(10, min(500, 20_000_000 // n)), dt=1e-2, temp=10 ** rng.uniform(-4, -2.5),
                 option=rng.choice(["plain", "plain", "damped", "walls"]))
    return c


# ---- inputs ------------------------------------------------------------------
def _packing(n, phi, radii, g):
    if radii == "bi":
        r = np.full(n, 0.5)
        r[:n // 2] = 0.7
    else:
        r = g.uniform(0.4, 0.6, n)
    box = math.sqrt(float(np.sum(r * r)) * math.pi / phi)
    return g.uniform(0.0, box, n), g.uniform(0.0, box, n), r, box


def _thermal(n, temp, g):
    vx, vy = g.normal(0.0, math.sqrt(temp), n), g.normal(0.0, math.sqrt(temp), n)
    return vx - vx.mean(), vy - vy.mean()


def _sizes(case):
    g = np.random.default_rng(case["pick"])
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [int(round(v)) for v in np.exp(g.uniform(lo, hi, case["systems"]))]


def _inputs(case, seed):
    """Host arrays of the case, from the seed alone."""
    g = np.random.default_rng(seed)
    if case["kind"] == "ens":
        return [_packing(n, case["phi"], "bi", g) for n in _sizes(case)]
    n = case["n"]
    if case["kind"] == "bumpy":
        x, y, r, box = _packing(n, case["phi"], "bi", g)
        nvb = np.where(r > 0.6, 28, 20).astype(np.int32)
        rv = bumpy_vertex_radius(1.0, 20, 0.9)
        vx, vy = _thermal(n, case["temp"], g)
        return dict(x=x, y=y, r=r, box=box, nvb=nvb, rv=rv, e_c=(2.0 * rv) ** 2, th=g.uniform(0, 2 * math.pi, n),
                    vx=vx, vy=vy, w=np.zeros(n))
    x, y, r, box = _packing(n, case["phi"], case["radii"], g)
    vx, vy = _thermal(n, case["temp"], g) if case["kind"] == "nve" else (np.zeros(n), np.zeros(n))
    return dict(x=x, y=y, vx=vx, vy=vy, r=r, m=np.ones(n), box=box)


KEYS = ("x", "y", "vx", "vy", "fx", "fy", "pe")


def prepare(case, seed):
    d = _inputs(case, seed)
    prec = dpg.MIXED if case["precision"] == "mixed" else dpg.FP64
    st = dict(case=case, stream=torch.cuda.Stream())
    if case["kind"] == "ens":
        st["data"] = [np.concatenate([s[k] for s in d]) for k in (0, 1, 2)]
        st["data"].append(np.ones(len(st["data"][0])))
        st["h"] = dpg.Ensemble([len(s[2]) for s in d], [s[3] for s in d], 1.7, 0.3, precision=prec)
    elif case["kind"] == "bumpy":
        st["data"] = d
        st["h"] = dpg.RigidBumpy(case["n"], int(d["nvb"].sum()), d["box"], d["e_c"], 2.0, d["rv"], 0.9, True,
                                 precision=prec)
    else:
        st["data"] = [torch.from_numpy(d[k]).cuda() for k in ("x", "y", "vx", "vy", "r", "m")]
        st["out"] = {k: torch.zeros(case["n"], dtype=torch.float64, device="cuda") for k in KEYS}
        torch.cuda.synchronize()
        st["h"] = dpg.Disk(case["n"], d["box"], precision=prec, stream=st["stream"].cuda_stream)
    return st


def run(st):
    case, h = st["case"], st["h"]
    kind = case["kind"]
    if kind == "ens":
        h.setState(*st["data"])
        res = h.minimizeFire(0.1, 1e-2, 0.0, 0.0, case["steps"], fmax_target=1e-13)
        out = h.getState()
        for k in ("avg_pe", "pressure", "contacts", "max_force"):
            out[k] = np.array([float(r[k]) for r in res])
        return out
    if kind == "bumpy":
        d = st["data"]
        h.setBodies(d["x"], d["y"], d["th"], d["r"], d["nvb"], d["vx"], d["vy"], d["w"])
        h.setMass(1.0)
        h.zeroForceAndPotentialEnergy()
        h.setupNeighbors(*BUMPY)
        if case["method"] == "nve":
            h.nveSteps(case["dt"], case["steps"])
        else:
            h.minimizeFire(0.1, 1e-2, 0.0, 0.0, case["steps"])
        out = h.getBodies()
        out["px"], out["py"] = h.getVertexPositions()
        return out
    ptrs = [C.cast(C.c_void_p(t.data_ptr()), DP) for t in st["data"]]
    check(h.lib.dpg_load_state(h.h, *ptrs, DEVICE))
    h.setupNeighbors(*(BI if case["radii"] == "bi" else POLY))
    out = dict(st["out"])
    if kind == "nve":
        if case["option"] == "damped":
            h.dampedNveSteps(case["dt"], 0.5, case["steps"])
        elif case["option"] == "walls":
            h.nveWallSteps(case["dt"], case["steps"])
        else:
            h.nveSteps(case["dt"], case["steps"])
    elif kind == "fire":
        r = dpg.minimizeFire(h, 0.1, 1e-2, 0.0, 0.0, case["steps"])
        out.update(avg_pe=r["avg_pe"], max_force=r["max_force"])
    else:
        h.zeroForceAndPotentialEnergy()
        h.calculateForces()
        out.update(pressure=h.getPressure(), contacts=h.getContactCount())
    h.getStateDevice(st["out"])
    torch.cuda.current_stream().wait_stream(st["stream"])
    return out


def work(case):
    """Inputs read and outputs written once; the state of a particle (position
    and velocity, read and written) again on every step where it does not fit
    on the chip; a contact's force and energy, about 30 operations, 2.5
    contacts a particle, and about 60 for its update."""
    if case["kind"] == "ens":
        n = sum(_sizes(case))
        per, steps = 64, case["steps"]
        if case["n_lo"] < 2048:
            steps = steps // 2  # the small systems converge before the cap
    elif case["kind"] == "bumpy":
        n, per, steps = case["n"], 24 * 16 + 180, case["steps"]
        return {"bytes": n * per, "flops": n * steps * (24 * 30 + 100)}
    else:
        n, per, steps = case["n"], 48 + 56, case.get("steps", 1)
    again = 64 * n * steps if n * 100 > 100e6 else 0
    return {"bytes": n * per + again, "flops": n * steps * (5 * 30 + 60)}


# ---- the same in 64 bits, plain torch --------------------------------------
def _image(d, box):
    return d - box * torch.round(d / box)


def _pairs(x, y, box, rc, own=None):
    """Directed pairs (i, j), i != j, closer than rc (own: not of one body)."""
    n, dev = len(x), x.device
    m = int(box // rc)
    out = []
    if m < 3:
        i, j = torch.meshgrid(torch.arange(n, device=dev), torch.arange(n, device=dev), indexing="ij")
        out.append((i.reshape(-1), j.reshape(-1)))
    else:
        cx = torch.floor(x / box * m).long() % m
        cy = torch.floor(y / box * m).long() % m
        cell = cx + cy * m
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=m * m)
        start = torch.cumsum(count, 0) - count
        table = torch.full((m * m, int(count.max())), -1, device=dev, dtype=torch.long)
        table[cell[order], torch.arange(n, device=dev) - start[cell[order]]] = order
        i0 = torch.arange(n, device=dev)
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                cand = table[(cx + ox) % m + ((cy + oy) % m) * m]
                keep = cand >= 0
                i, j = i0[:, None].expand_as(cand)[keep], cand[keep]
                d2 = _image(x[i] - x[j], box) ** 2 + _image(y[i] - y[j], box) ** 2
                near = d2 < rc * rc
                out.append((i[near], j[near]))
    i, j = torch.cat([a for a, _ in out]), torch.cat([b for _, b in out])
    keep = i != j if own is None else own[i] != own[j]
    return i[keep], j[keep]


class _Field:
    """Harmonic contacts of disks, with a list that is renewed as they move."""

    def __init__(self, r, box, e_c=1.0, own=None):
        self.r, self.box, self.e_c, self.own, self.ref = r, box, e_c, own, None
        self.d = 2.0 * float(r.max())
        self.skin = 0.25 * self.d

    def __call__(self, x, y):
        if self.ref is None or float(((x - self.ref[0]) ** 2 + (y - self.ref[1]) ** 2).max()) > (self.skin / 2) ** 2:
            self.ref = (x.clone(), y.clone())
            self.i, self.j = _pairs(x, y, self.box, self.d + self.skin, self.own)
        i, j = self.i, self.j
        dx, dy = _image(x[i] - x[j], self.box), _image(y[i] - y[j], self.box)
        rs, d2 = self.r[i] + self.r[j], dx * dx + dy * dy
        hit = (d2 < rs * rs).nonzero()[:, 0]
        i, dx, dy, rs = i[hit], dx[hit], dy[hit], rs[hit]
        d = torch.sqrt(d2[hit])
        ov = 1.0 - d / rs
        fm = self.e_c * ov / (rs * d)
        z = torch.zeros_like(x)
        self.hits = len(hit)
        self.virial = float((fm * d * d).sum())
        return (z.index_add(0, i, fm * dx), z.index_add(0, i, fm * dy), z.index_add(0, i, 0.25 * self.e_c * ov * ov))


def _walls(x, y, r, box):
    fx, fy, pe = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
    for p, f in ((x, fx), (y, fy)):
        for dist, sign in ((p, 1.0), (box - p, -1.0)):
            ov = torch.clamp(r - dist, min=0.0)
            f += sign * ov / (r * r)
            pe += 0.5 * (ov / r) ** 2
    return fx, fy, pe


def _fire(move, kick, mix, force, steps):
    """FIRE as the library runs it: move(dt), kick(dt), mix(alpha), force() -> power."""
    dt, alpha, good, bad = 1e-2, 0.1, 0, 0
    power = force()
    for _ in range(steps):
        if power > 0:
            good, bad = good + 1, 0
            if good > 5:
                dt, alpha = min(dt * 1.1, 0.1), alpha * 0.99
            up = False
        else:
            good, bad = 0, bad + 1
            if bad > 10:
                break
            dt, alpha, up = max(dt * 0.5, 1e-5), 0.1, True
        if up:
            move(-dt / 2, True)
        kick(dt / 2)
        mix(alpha)
        move(dt, False)
        force()
        kick(dt / 2)
        power = force(True)


def _mixed_v(v, f, alpha):
    vn, fn = torch.sqrt(v[0] ** 2 + v[1] ** 2), torch.sqrt(f[0] ** 2 + f[1] ** 2)
    on = fn > 1e-16
    m = torch.where(on, vn / torch.where(on, fn, torch.ones_like(fn)) * alpha, torch.zeros_like(fn))
    return [torch.where(on, u, torch.zeros_like(u)) * (1 - alpha) + g * m for u, g in zip(v, f)]


def _disk_fire(x, y, r, box, steps):
    field = _Field(r, box)
    s = dict(x=x.clone(), y=y.clone(), v=[torch.zeros_like(x), torch.zeros_like(x)])

    def force(known=False):
        if not known:
            s["fx"], s["fy"], s["pe"] = field(s["x"], s["y"])
        return float((s["fx"] * s["v"][0] + s["fy"] * s["v"][1]).sum())

    def move(dt, stop):
        s["x"], s["y"] = s["x"] + s["v"][0] * dt, s["y"] + s["v"][1] * dt
        if stop:
            s["v"] = [torch.zeros_like(x), torch.zeros_like(x)]

    def kick(dt):
        s["v"] = [s["v"][0] + s["fx"] * dt, s["v"][1] + s["fy"] * dt]

    def mix(alpha):
        s["v"] = _mixed_v(s["v"], (s["fx"], s["fy"]), alpha)

    _fire(move, kick, mix, force, steps)
    s["field"] = field
    return s


def _fmax(s):
    return float(torch.sqrt(s["fx"] ** 2 + s["fy"] ** 2).max())


def _exact_ens(case, seed):
    if case["steps"] > 400:  # FP32 trajectories have parted from any other rounding's by then
        return None
    got = {k: [] for k in ("x", "y", "fx", "fy")}
    per = {k: [] for k in ("avg_pe", "pressure", "contacts", "max_force")}
    for x, y, r, box in _inputs(case, seed):
        x, y, r = (torch.from_numpy(a).cuda() for a in (x, y, r))
        s = _disk_fire(x, y, r, box, case["steps"])
        for k in got:
            got[k].append(s[k])
        per["avg_pe"].append(float(s["pe"].mean()))
        per["pressure"].append(s["field"].virial / (4.0 * box * box))
        per["contacts"].append(float(s["field"].hits))
        per["max_force"].append(_fmax(s))
    out = {k: torch.cat(v) for k, v in got.items()}
    out.update({k: np.array(v) for k, v in per.items()})
    out["pressure"] = None  # reported by jamming runs only
    return out


def _exact_bumpy(case, seed):
    d = _inputs(case, seed)
    t = {k: torch.from_numpy(np.asarray(v)).cuda() for k, v in d.items() if isinstance(v, np.ndarray)}
    n, box, rv = case["n"], d["box"], d["rv"]
    own = torch.repeat_interleave(torch.arange(n, device="cuda"), t["nvb"].long())
    first = torch.cumsum(t["nvb"].long(), 0) - t["nvb"].long()
    k = torch.arange(len(own), device="cuda") - first[own]
    a = k * (2 * math.pi / t["nvb"].double())[own] + t["th"][own]
    arm = (t["r"] - rv)[own]
    qx, qy = arm * torch.cos(a), arm * torch.sin(a)
    inertia = (t["r"] - rv) ** 2
    field = _Field(torch.full((len(own),), rv, device="cuda", dtype=torch.float64), box, d["e_c"], own)
    s = dict(x=t["x"], y=t["y"], th=t["th"], qx=qx, qy=qy)
    fire = case["method"] == "fire"
    zero = torch.zeros_like(t["x"])
    s["v"], s["w"] = ([zero, zero], zero) if fire else ([t["vx"], t["vy"]], t["w"])

    def force(known=False):
        if not known:
            fx, fy, pe = field(s["x"][own] + s["qx"], s["y"][own] + s["qy"])
            s["fx"], s["fy"], s["pe"] = (zero.index_add(0, own, u) for u in (fx, fy, pe))
            s["tq"] = zero.index_add(0, own, fy * s["qx"] - fx * s["qy"])
        return float((s["fx"] * s["v"][0] + s["fy"] * s["v"][1] + s["tq"] * s["w"]).sum())

    def move(dt, stop):
        s["x"], s["y"] = s["x"] + s["v"][0] * dt, s["y"] + s["v"][1] * dt
        da = s["w"] * dt
        c, e = torch.cos(da)[own], torch.sin(da)[own]
        s["th"] = s["th"] + da
        s["qx"], s["qy"] = s["qx"] * c - s["qy"] * e, s["qx"] * e + s["qy"] * c
        if stop:
            s["v"], s["w"] = [zero, zero], zero

    def kick(dt):
        s["v"] = [s["v"][0] + s["fx"] * dt, s["v"][1] + s["fy"] * dt]
        s["w"] = s["w"] + s["tq"] * dt / inertia

    def mix(alpha):
        s["v"] = _mixed_v(s["v"], (s["fx"], s["fy"]), alpha)
        on = s["tq"].abs() > 1e-16
        m = torch.where(on, s["w"].abs() / torch.where(on, s["tq"].abs(), torch.ones_like(zero)) * alpha, zero)
        s["w"] = torch.where(on, s["w"], zero) * (1 - alpha) + s["tq"] * m

    if fire:
        _fire(move, kick, mix, force, case["steps"])
        s["v"], s["w"] = [zero, zero], zero
    else:
        dt = case["dt"]
        force()
        for _ in range(case["steps"]):
            kick(dt / 2)
            move(dt, False)
            force()
            kick(dt / 2)
    out = {k: s[k] for k in ("x", "y", "th", "w", "fx", "fy", "tq", "pe")}
    out.update(vx=s["v"][0], vy=s["v"][1], I=inertia, px=s["x"][own] + s["qx"], py=s["y"][own] + s["qy"])
    return out


def exact(case, seed):
    if case["kind"] == "ens":
        return _exact_ens(case, seed)
    if case["kind"] == "bumpy":
        return _exact_bumpy(case, seed)
    d = _inputs(case, seed)
    x, y, vx, vy, r = (torch.from_numpy(d[k]).cuda() for k in ("x", "y", "vx", "vy", "r"))
    box = d["box"]
    if case["kind"] == "fire":
        s = _disk_fire(x, y, r, box, case["steps"])
        out = {k: s[k] for k in ("x", "y", "fx", "fy", "pe")}
        out.update(vx=torch.zeros_like(x), vy=torch.zeros_like(x), avg_pe=float(s["pe"].mean()), max_force=_fmax(s))
        return out
    field = _Field(r, box)
    fx, fy, pe = field(x, y)
    out = {}
    if case["kind"] == "nve":
        dt, opt = case["dt"], case["option"]
        for _ in range(case["steps"]):
            vx, vy = vx + fx * (dt / 2), vy + fy * (dt / 2)
            x, y = x + vx * dt, y + vy * dt
            fx, fy, pe = field(x, y)
            if opt == "damped":
                fx, fy = fx - 0.5 * vx, fy - 0.5 * vy
            elif opt == "walls":
                wx, wy, we = _walls(x, y, r, box)
                fx, fy, pe = fx + wx, fy + wy, pe + we
            vx, vy = vx + fx * (dt / 2), vy + fy * (dt / 2)
    else:
        out.update(pressure=field.virial / (4.0 * box * box), contacts=float(field.hits))
    out.update(x=x, y=y, vx=vx, vy=vy, fx=fx, fy=fy, pe=pe)
    return out
