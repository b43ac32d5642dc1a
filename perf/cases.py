"""Timed cases of the explicit MPM step: what a user of the framework runs.

Each case is one output interval of a simulation through the public Python
binding: a number of steps, then the particle fields and scalars that a host
program reads back for its result files. The mixed form (batched engine,
single scene or served scenes) and the two FP64 forms are covered with every
shape family and step scheme, from a few thousand particles (launch-bound)
to several millions (device-bound).

The mixed form's particle interpolants and stresses are single precision, so
its results are returned as float32 (displacements in place of positions,
whose size would hide them); everything of the FP64 forms is float64.

exact() restates the step in plain torch float64 (linear, GIMP, B-spline and
SGMP shapes; elastic, Drucker-Prager, neo-Hookean and null materials).
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "mpm3d-f90_gb300"))

import mpm3d_gb300 as mpm  # noqa: E402

# the routines of one MUSL step, in the order of the reference's time loop
PHASES_MUSL = ("BeginStep", "GridMomentumInitial", "GridMomentumUpdate", "IntegrateMomentum",
               "ParticlePositionUpdate", "GridMomentumMUSL", "ApplyBoundaryConditions",
               "ParticleStressUpdate", "calcEnergy", "UpdateDT", "SmoothStressbyGrid")


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the shipped Cook-membrane example at its published resolution (5776
        # particles), SGMP, smoothed pressure read with each frame: the
        # smallest calls, where launches count
        dict(name="cook-6k-mixed", kind="cook", dp=0.5, shape="sgmp", form="mixed", steps=40),
        # an elastic block thrown onto a floor, linear grid, odd counts
        dict(name="block-36k-mixed", kind="block", n=33, shape="linear", scheme="musl", form="mixed", steps=50),
        # soil slope at 0.2 m and at the benchmark's 0.1 m spacing (GIMP, USF)
        dict(name="slope-150k-mixed", kind="slope", dp=0.2, width=3.0, form="mixed", steps=50),
        dict(name="slope-1200k-mixed", kind="slope", dp=0.1, width=3.0, form="mixed", steps=50),
        # dam break at 2 cm spacing (quadratic B-spline, MUSL, null material)
        dict(name="dam-2000k-mixed", kind="dam", dp=0.02, form="mixed", steps=40),
        # granular column collapse, the largest scene (GIMP, MUSL)
        dict(name="column-4100k-mixed", kind="column", scale=2.5, form="mixed", steps=40),
        # soft cantilever, neo-Hookean, SGMP, MUSL
        dict(name="beam-95k-mixed", kind="beam", n=25, form="mixed", steps=50),
        # the serving runtime: twelve scenes of uneven size submitted at once,
        # 60 steps each, every scene's velocities and stresses fetched
        dict(name="serve-12-mixed", kind="serve", scenes=12, smallest=2500, largest=250000, steps=60),
        # the plain FP64 forms: the Taylor bar (Johnson-Cook, linear, USF) and
        # the soil slope in the strict form, the dam break in the native form
        dict(name="bar-17k-fp64", kind="bar", dp=4e-4, form="fp64", steps=20),
        dict(name="slope-150k-fp64", kind="slope", dp=0.2, width=3.0, form="fp64", steps=8),
        dict(name="dam-31k-native", kind="dam", dp=0.08, form="native", steps=10),
        # the drop-in boundary: a host time loop that calls one routine per
        # phase and reads the scalars every step, as the Fortran program does
        dict(name="cook-6k-host", kind="cook", dp=0.5, shape="gimp", form="fp64", steps=15, host=True),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    """A case of the same ranges: a workload, a size (logarithmic) and a form."""
    kind = rng.choice(["cook", "block", "slope", "slope", "dam", "dam", "column", "beam", "serve", "bar"])
    form = rng.choice(["mixed", "mixed", "mixed", "fp64", "native"])
    if kind == "cook":
        shape = rng.choice(["mpm", "gimp", "bimp", "sgmp"])
        return dict(kind="cook", dp=round(_log(rng, 0.25, 0.9), 3), shape=shape, form=form,
                    steps=rng.randrange(15, 45), host=form != "mixed" and rng.random() < 0.5)
    if kind == "block":
        return dict(kind="block", n=rng.randrange(11, 101 if form == "mixed" else 42), shape=rng.choice(["linear", "gimp", "bimp"]),
                    scheme=rng.choice(["usf", "musl"]), form=form, steps=rng.randrange(20, 60) if form == "mixed" else rng.randrange(5, 12))
    if kind == "slope":
        if form == "mixed":
            return dict(kind="slope", dp=round(_log(rng, 0.1, 0.5), 3), width=3.0, form=form, steps=rng.randrange(20, 60))
        return dict(kind="slope", dp=round(_log(rng, 0.18, 0.5), 3), width=3.0, form=form, steps=rng.randrange(4, 10))
    if kind == "dam":
        if form == "mixed":
            return dict(kind="dam", dp=round(_log(rng, 0.018, 0.1), 4), form=form, steps=rng.randrange(20, 50))
        return dict(kind="dam", dp=round(_log(rng, 0.05, 0.12), 4), form=form, steps=rng.randrange(4, 10))
    if kind == "column":
        return dict(kind="column", scale=round(_log(rng, 2.6, 10.0), 3), form="mixed", steps=rng.randrange(15, 40))
    if kind == "beam":
        return dict(kind="beam", n=rng.randrange(9, 41), form="mixed", steps=rng.randrange(20, 60))
    if kind == "serve":
        lo = int(_log(rng, 2000, 9000))
        return dict(kind="serve", scenes=rng.randrange(5, 17), smallest=lo, largest=int(_log(rng, 30000, 250000)),
                    steps=rng.randrange(30, 70))
    return dict(kind="bar", dp=round(_log(rng, 3e-4, 8e-4), 6), form=rng.choice(["fp64", "native"]), steps=rng.randrange(8, 24))


# ------------------------------------------------------------------ scenes
def _f(x):
    return float(np.float32(x))


def _s(x):
    return "%.9g" % _f(x)


def _cells(length, h):
    """The length rounded up to whole cells."""
    return h * math.ceil(length / h - 1e-6)


def _points(mass, xyz):
    m = _s(mass)
    p = np.asarray(xyz, dtype=np.float32).tolist()
    return "\n".join(["part poin 1 %d" % len(p)] +
                     ["%d 1 %s %.9g %.9g %.9g" % (i + 1, m, a, b, c) for i, (a, b, c) in enumerate(p)])


def _scene(c, seed):
    """A scene: its deck (reference syntax) and the same data as plain values
    for exact()."""
    r = np.random.default_rng(seed)
    k = c["kind"]
    s = dict(grav=(0.0, 0.0, 0.0), vel=(0.0, 0.0, 0.0), loads=None, qload=0.0, damp=0.0, bq=(_f(1.5), _f(0.06)), bodies=1)
    if k == "slope":  # 45 degree slope on a rigid base, jittered lattice, Drucker-Prager
        dp, w, H = c["dp"], c["width"], 20.0
        h = 2 * dp
        nx, ny, nz = int(round(30.0 / dp)), 2 * int(round(w / h)), int(round(H / dp))  # whole cells between the side walls
        X, Z = np.meshgrid((np.arange(nx) + 0.5) * dp, (np.arange(nz) + 0.5) * dp)
        keep = Z < np.where(X <= 10.0, H, H - (X - 10.0))
        xs, zs = X[keep], Z[keep]
        xyz = np.concatenate([np.stack([xs, np.full(xs.shape, (j + 0.5) * dp), zs], axis=1) for j in range(ny)])
        xyz = (xyz + r.uniform(-0.01 * dp, 0.01 * dp, size=xyz.shape)).astype(np.float32)
        t = math.tan(math.radians(20.0))
        q, kk = 3 * t / math.sqrt(9 + 12 * t * t), 3e4 / math.sqrt(9 + 12 * t * t)
        s.update(h=h, span=((0.0, _cells(36.0, h)), (0.0, ny * dp), (0.0, _cells(24.0, h))), dtsc=0.3, scheme="usf", shape="gimp",
                 fix=(2, 0, 2, 2, 1, 0), mat=("dpm", 2000.0, 5e7, 0.3, q, kk, 0.0, kk / q), mass=2000.0 * dp ** 3,
                 parts=("poin", xyz), grav=(0.0, 0.0, -9.81))
    elif k == "dam":  # water column in a tank with slip walls, released from rest
        dp = c["dp"]
        h = 2 * dp
        n = [int(round(v / dp)) for v in (4.0, 2.0, 2.0)]
        # the walls on grid lines: the tank is a whole number of cells
        tank = [_cells(v, h) for v in (10.0, max(2.0, n[1] * dp), 4.0)]
        s.update(h=h, span=tuple((-h, t + h) for t in tank), dtsc=0.5, scheme="musl", shape="bimp", fix=(2, 2, 2, 2, 2, 0),
                 mat=("null", 1000.0, 2.2e6 * r.uniform(0.9, 1.1), 1e-3), rho=1000.0,
                 parts=("bloc", dp, (0.0, 0.0, 0.0), n), grav=(0.0, 0.0, -9.81))
    elif k == "column":  # cylinder of sand on a rough floor
        sc = c["scale"]
        dp = _f(2.307e-3 * sc)
        t = math.tan(math.radians(r.uniform(28.0, 32.0)))
        nl, nr = int(round(1.0 / dp)), int(round(0.5 / dp))
        h = 4e-3 * sc
        half = _cells(1.024, h)
        s.update(h=h, span=((-half, half), (-half, half), (0.0, half)), dtsc=0.5, scheme="musl", shape="gimp",
                 fix=(0, 0, 0, 0, 1, 0), mat=("dpm", 2650.0, 1e7 * r.uniform(0.9, 1.1), 0.3, 3 * t / math.sqrt(9 + 12 * t * t), 0.0, 0.0, 0.0),
                 rho=2650.0, parts=("cicl", dp, nl, nr), grav=(0.0, 0.0, -9.81), bodies=nl)
    elif k == "beam":  # 6 x 1 x 1 m cantilever, clamped at x = 0, n particles through the depth
        n = c["n"]
        dp = 1.0 / n
        h, z0 = 2 * dp, 2.0
        s.update(h=h, span=((-h, _cells(8.0, h)), (-h, _cells(n * dp, h) + h), (0.0, _cells(z0 + n * dp, h) + 2 * h)), dtsc=0.5, scheme="musl", shape="sgmp",
                 fix=(1, 0, 2, 2, 0, 0), mat=("neoh", 1000.0, r.uniform(1.5e7, 6e7), r.uniform(0.3, 0.45)), rho=1000.0,
                 parts=("bloc", dp, (0.0, 0.0, z0), (6 * n, n, n)), grav=(0.0, 0.0, -9.81))
    elif k == "block":  # an elastic cube thrown onto the floor
        n, dp, h = c["n"], 0.5, 1.0
        L = n * dp
        s.update(h=h, span=((-8 * h, math.ceil(L) + 8 * h), (-8 * h, math.ceil(L) + 8 * h), (-h, math.ceil(L) + 10 * h)),
                 dtsc=0.4, scheme=c["scheme"], shape=c["shape"], fix=(0, 0, 0, 0, 2, 0),
                 mat=("elas", 1000.0, 1e7 * r.uniform(0.8, 1.2), 0.3), rho=1000.0,
                 parts=("bloc", dp, (0.1, 0.2, 0.0), (n, n, n)), grav=(0.0, 0.0, -9.81),
                 vel=(r.uniform(-1, 1), r.uniform(-1, 1), -5.0))
    elif k == "cook":  # Cook's tapered panel, sheared at x = 48, quasi-static
        ds = c["dp"]
        xs = (np.arange(int(round(48 / ds))) + 0.5) * ds
        ys = (np.arange(int(round(60 / ds))) + 0.5) * ds
        Y, X = np.meshgrid(ys, xs, indexing="ij")
        keep = (Y >= 44.0 / 48.0 * X) & (Y <= 44.0 + 16.0 / 48.0 * X)
        xyz = np.stack([X[keep], Y[keep], np.zeros(int(keep.sum()))], axis=1).astype(np.float32)
        n, h = len(xyz), 2 * ds
        z = h / 2 if c["shape"] in ("mpm", "sgmp") else h
        # one cell thick under SGMP: the mid-plane stays clear of the half cell
        # (a tie between the two node layers) unless h / 2 is exact
        dz = h / 64 if c["shape"] == "sgmp" and math.frexp(_f(h))[0] != 0.5 else 0.0
        lo = 0.0 if c["shape"] == "mpm" else -h
        right = np.where(np.isclose(xyz[:, 0], np.float32(xs[-1])))[0]
        per = r.uniform(0.9, 1.1) / max(1, len(right) - 1)
        f = np.array([_f(per * (0.5 if j in (0, len(right) - 1) else 1.0)) for j in range(len(right))])
        s.update(h=h, span=((lo, lo + h * math.ceil((50 - lo) / h)), (lo, lo + h * math.ceil((62 - lo) / h)), (-z - dz, z - dz)), dtsc=0.8,
                 scheme="musl", shape="linear" if c["shape"] == "mpm" else c["shape"], fix=(1, 0, 0, 0, 2, 2),
                 mat=("neoh", 1.0, 70.0 * r.uniform(0.9, 1.1), 0.45), mass=1440.0 / n, parts=("poin", xyz),
                 loads=(right, 1, f), qload=15.0, damp=0.3, smooth=True)
    elif k == "bar":  # copper cylinder thrown onto a rigid wall, Johnson-Cook with failure
        dp, rad = c["dp"], 3.2e-3
        n = int(math.ceil(rad / dp))
        X, Y = np.meshgrid((np.arange(-n, n) + 0.5) * dp, (np.arange(-n, n) + 0.5) * dp)
        ins = X ** 2 + Y ** 2 < rad ** 2
        xyz = np.concatenate([np.stack([X[ins], Y[ins], np.full(int(ins.sum()), (j + 0.5) * dp)], axis=1)
                              for j in range(int(round(32.4e-3 / dp)))]).astype(np.float32)
        h = 2 * dp
        half = _cells(2.0 * rad, h)
        K = 1.17e11 / (3 * (1 - 0.7))
        s.update(h=h, span=((-half, half), (-half, half), (0.0, _cells(40e-3, h))), dtsc=0.1, scheme="usf", shape="linear",
                 fix=(0, 0, 0, 0, 1, 0), mat=("jcf", 8930.0, 1.17e11, 0.35, 9e7, 2.92e8, 0.31, 0.025, 1.09, 293, 1356, 383, 1, 100.0),
                 eos="seos 1 1 0 %s 0 0 0 0 0 0" % _s(K), mass=8930.0 * dp ** 3, parts=("poin", xyz),
                 vel=(0.0, 0.0, -190.0 * r.uniform(0.95, 1.05)))
    else:
        raise ValueError(k)
    kind = s["parts"][0]
    if kind == "poin":
        np_, body = len(s["parts"][1]), [_points(s["mass"], s["parts"][1])]
    elif kind == "bloc":
        _, dp, o, n = s["parts"]
        np_ = n[0] * n[1] * n[2]
        body = ["part bloc 1 1 %s %s %s %s %s %d %d %d" % (_s(s["rho"]), _s(dp), _s(o[0]), _s(o[1]), _s(o[2]), *n)]
    else:
        _, dp, nl, nr = s["parts"]
        np_ = len(_disc(dp, nr)) * nl
        body = ["part cicl 1 1 %s %s 0 0 %s %d" % (_s(s["rho"]), _s(dp), _s(j * dp), nr) for j in range(nl)]
    d = ["mpm3d *** %s" % k, "nbco 1", "nbbo %d" % s["bodies"], "nbmp %d" % np_, "nmat 1"]
    d += ["%s %s %s" % (key, _s(a), _s(b)) for key, (a, b) in zip(("spx", "spy", "spz"), s["span"])]
    d += ["dcel %s" % _s(s["h"]), "dtsc %s" % _s(s["dtsc"]), "endt 1000.0", "%s on" % s["scheme"]]
    if s["shape"] != "linear":
        d.append(s["shape"])
    d.append("fixe %d %d %d %d %d %d" % s["fix"])
    if s["qload"]:
        d += ["QuLo %s" % _s(s["qload"]), "Damp %s" % _s(s["damp"])]
    if s.get("smooth"):
        d.append("smoo")
    m = s["mat"]
    d += ["mate", "1 %s %s" % (m[0], " ".join(_s(v) for v in m[1:]))]
    if m[0] == "null":
        d.append("seos 1 4 %s" % _s(math.sqrt(_f(m[2]) / _f(m[1]))))
    if "eos" in s:
        d.append(s["eos"])
    d += body
    if any(s["vel"]):
        d += ["velo", "body 1 %s %s %s" % tuple(_s(v) for v in s["vel"]), "endv"]
    if any(s["grav"]) or s["loads"]:
        d.append("load")
        d += ["grav %d %s %s %s" % (b + 1, *(_s(v) for v in s["grav"])) for b in range(s["bodies"] if any(s["grav"]) else 0)]
        if s["loads"]:
            d += ["part %d 0 %s 0" % (i + 1, _s(f)) for i, f in zip(s["loads"][0], s["loads"][2])]
        d.append("endl")
    s.update(np=np_, deck="\n".join(d + ["endi"]) + "\n")
    return s


def _disc(dp, nr):
    """Positions of one layer of the disc generator, in its order."""
    t = (np.arange(1 - nr, nr + 1, dtype=np.float64) - 1) * dp + 0.5 * dp
    A, B = np.meshgrid(t, t, indexing="ij")
    keep = A * A + B * B < (nr * dp) ** 2
    return np.stack([A[keep], B[keep]], axis=1)


def _particles(s):
    """Positions [3, n] and mass [n] of a scene, in deck order (float64)."""
    kind = s["parts"][0]
    if kind == "poin":
        x = s["parts"][1].astype(np.float64).T
        return np.ascontiguousarray(x), np.full(x.shape[1], _f(s["mass"]))
    if kind == "bloc":
        _, dp, o, n = s["parts"]
        dp = _f(dp)
        ax = [np.arange(n[a], dtype=np.float64) * dp + (_f(o[a]) + dp * 0.5) for a in range(3)]
        Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        x = np.stack([X.ravel(), Y.ravel(), Z.ravel()])
    else:
        _, dp, nl, nr = s["parts"]
        dp = _f(dp)
        one = _disc(dp, nr)
        x = np.empty((3, nl * len(one)))
        x[0], x[1] = np.tile(one[:, 0], nl), np.tile(one[:, 1], nl)
        x[2] = np.repeat([_f(j * dp) + dp * 0.5 for j in range(nl)], len(one))
    return x, np.full(x.shape[1], _f(s["rho"]) * dp ** 3)


def _served(c, seed):
    """The scenes of a serving case: sizes spread logarithmically, panels and
    beams alternating, their stiffness from the seed."""
    n = c["scenes"]
    out = []
    for i in range(n):
        target = c["smallest"] * (c["largest"] / c["smallest"]) ** (i / (n - 1))
        if i % 2:
            out.append(_scene(dict(kind="cook", dp=round(math.sqrt(1440.0 / min(target, 60000)), 4), shape="sgmp"), seed * 64 + i))
        else:
            out.append(_scene(dict(kind="beam", n=max(5, int(round((target / 6.0) ** (1.0 / 3.0))))), seed * 64 + i))
    return out


# ------------------------------------------------------------ prepare / run
FIELDS = (("Xp", 3), ("VXp", 3), ("SM", 1), ("SD", 6))


def prepare(case, seed):
    if case["kind"] == "serve":
        decks = [mpm.Deck.parse(s["deck"]) for s in _served(case, seed)]
        return dict(case=case, server=mpm.Server(policy="fifo"), decks=decks)
    s = _scene(case, seed)
    deck = mpm.Deck.parse(s["deck"])
    ctx = mpm.MpmStep(deck, case["form"])
    out = {f: mpm.pinned_empty(nc * s["np"]) for f, nc in FIELDS + ((("Spre", 1),) if s.get("smooth") else ())}
    x0 = torch.from_numpy(deck.particles()["Xp"].reshape(-1)) if case["form"] == "mixed" else None
    return dict(case=case, ctx=ctx, deck=deck, out=out, x0=x0)


def _single(a):
    return torch.from_numpy(np.asarray(a)).to(torch.float32)


def run(state):
    c = state["case"]
    if c["kind"] == "serve":
        srv = state["server"]
        tickets = [srv.submit(d, c["steps"], fields=("VXp", "SD")) for d in state["decks"]]
        out = []
        for t in tickets:
            srv.wait(t)
            out.append([_single(srv.field(t, "VXp")), _single(srv.field(t, "SD"))])
            srv.release(t)
        return out
    ctx = state["ctx"]
    if c.get("host"):
        for _ in range(c["steps"]):
            for ph in PHASES_MUSL:
                ctx.phase(ph)
            sc = ctx.scalars()  # the loop's exit test and report read these
    else:
        ctx.run(c["steps"])
        sc = ctx.scalars()
    out = {f: ctx.download(f, out=b) for f, b in state["out"].items()}
    tot = np.array([sc[k] for k in ("CurrentTime", "DT", "EngKinetic", "EngInternal", "Momentum_x", "Momentum_y", "Momentum_z")])
    out["istep"], out["totals"] = int(sc["istep"]), tot
    if c["form"] == "mixed":
        x = torch.from_numpy(np.asarray(out.pop("Xp")).reshape(-1)) - state["x0"]
        out = {f: v if f == "istep" else _single(v) for f, v in out.items()}
        out["disp"] = x.to(torch.float32).reshape(3, -1)
    return out


def work(case):
    """Bytes: every particle field a step must read and write once, at the
    form's widths, the active nodes' data (one node per 8 particles), and the
    fields returned. Flops: the shape-function transfers of a step."""
    if case["kind"] == "serve":
        scenes = [(s["np"], s) for s in _served(case, 1)]
    else:
        s = _scene(case, 1)
        scenes = [(s["np"], s)]
    total = flops = 0.0
    for n, s in scenes:
        f64 = case.get("form") in ("fp64", "native")
        b = 8 if f64 else 4
        per = 2 * (24 + 24 + 8) + 8 + b * 20  # x, v, ie read and written, mass; volume, stresses, q, cp
        per += {"dpm": 2 * b, "neoh": 18 * b, "jcf": 6 * b}.get(s["mat"][0], 0)
        per += (160.0 if s["scheme"] == "musl" else 112.0) / 8
        nodes = {"linear": 8, "gimp": 12, "bimp": 27, "sgmp": 8}[s["shape"]]
        total += n * (case["steps"] * per + (12 * b + 3 * 8))
        flops += n * case["steps"] * (nodes * (70 if s["scheme"] == "musl" else 62) + 150)
    return {"bytes": total, "flops": flops}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    if case["kind"] == "bar":
        return None  # Johnson-Cook: an increment is carried from particle to particle in processing order
    if case["kind"] == "serve":
        out = []
        for s in _served(case, seed):
            r = _reference(s, case["steps"])
            out.append([r["VXp"], r["SD"]])
        return out
    s = _scene(case, seed)
    r = _reference(s, case["steps"])
    r["istep"], r["totals"] = None, None
    if case["form"] == "mixed":
        x = r.pop("Xp")
        r["disp"] = x - torch.from_numpy(_particles(s)[0]).to(x.device)
    if s.get("smooth"):
        r["Spre"] = None
    return r


_CORNERS = [(i, j, k) for k in (0, 1) for j in (0, 1) for i in (0, 1)]


def _weights(shape, x, s0, h, NG):
    """Per direction: node indices, weights and derivatives (lists over the
    nodes of the direction; a node off the grid has weight 0)."""
    out = []
    for a in range(3):
        u = (x[a] - s0[a]) / h
        c = torch.floor(u)
        o = u - c
        if shape == "linear":
            tab = [(0, 1 - o, -torch.ones_like(o)), (1, o, torch.ones_like(o))]
        elif shape == "bimp":
            tab = [(-1, 0.5 * (1 - o) ** 2, o - 1), (0, 0.5 + o - o * o, 1 - 2 * o), (1, 0.5 * o * o, o)]
        else:
            tab = []
            for t in (-1, 0, 1, 2):
                r = o - t
                b, sg = r.abs(), torch.sign(r)
                w = torch.where(b < 0.25, (7 - 16 * b * b) / 8,
                                torch.where(b < 0.75, 1 - b, torch.where(b < 1.25, ((5 - 4 * b) / 4) ** 2, torch.zeros_like(b))))
                d = torch.where(b < 0.25, -4 * r,
                                torch.where(b < 0.75, -sg, torch.where(b < 1.25, 2 * r - 2.5 * sg, torch.zeros_like(b))))
                tab.append((t, w, d))
        rows = []
        for t, w, d in tab:
            n = c.long() + t
            ok = (n >= 0) & (n < NG[a])
            rows.append((n.clamp(0, NG[a] - 1), w * ok, d * ok / h))
        out.append(rows)
    return out


def _slots(wt, NG):
    """(flat node, weight, (dx, dy, dz)) for every node of the box."""
    for nz, wz, dz in wt[2]:
        for ny, wy, dy in wt[1]:
            row = (nz * NG[1] + ny) * NG[0]
            wyz, dwy, dwz = wy * wz, dy * wz, wy * dz
            for nx, wx, dx in wt[0]:
                yield row + nx, wx * wyz, (dx * wyz, wx * dwy, wx * dwz)


def _reference(s, steps):
    """The explicit step (USF / USL / MUSL) in float64."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    F = torch.float64
    xa, ma = _particles(s)
    x, m = torch.from_numpy(xa).to(dev), torch.from_numpy(ma).to(dev)
    n = x.shape[1]
    h = _f(s["h"])
    s0 = [_f(a) for a, _ in s["span"]]
    NC = [int((_f(b) - _f(a)) / h + 0.5) for a, b in s["span"]]
    NG = [v + 1 for v in NC]
    nn, ncell = NG[0] * NG[1] * NG[2], NC[0] * NC[1] * NC[2]
    name, sg = s["mat"][0], s["shape"] == "sgmp"
    mp = [_f(v) for v in s["mat"][1:]]
    rho = mp[0]
    cutoff = rho * h ** 3 * float(np.float32(1e-5))
    if name == "null":
        c0 = math.sqrt(mp[1] / rho)
        wave = cp0 = c0
        E = nu = 0.0
    else:
        E, nu = mp[1], mp[2]
        wave = math.sqrt(E * (1 - nu) / (1 + nu) / (1 - 2 * nu) / rho)
        cp0 = wave if name in ("elas", "neoh") else 0.0
    G2, lam, K3 = E / (1 + nu), E * nu / ((1 + nu) * (1 - 2 * nu)), E / (1 - 2 * nu)
    v = torch.tensor([_f(a) for a in s["vel"]], dtype=F, device=dev)[:, None].repeat(1, n)
    fxp = torch.zeros(3, n, dtype=F, device=dev)
    if s["loads"]:
        fxp[s["loads"][1], torch.from_numpy(s["loads"][0]).to(dev)] = torch.from_numpy(s["loads"][2]).to(dev)
    grav = torch.tensor([_f(a) for a in s["grav"]], dtype=F, device=dev)[:, None]
    z = lambda *k: torch.zeros(*k, n, dtype=F, device=dev)  # noqa: E731
    vol, sm, sd, q, H = m / rho, z(), z(6), z(), z(3, 3)  # sd: xx yy zz xy yz xz
    # fixities: the outer node layer, two layers for GIMP, B-spline and SGMP
    idx = torch.arange(nn, device=dev)
    ij = (idx % NG[0], idx // NG[0] % NG[1], idx // (NG[0] * NG[1]))
    two = 0 if s["shape"] == "linear" else 1
    fixed = torch.zeros(3, nn, dtype=torch.bool, device=dev)
    bdt = torch.zeros(3, nn, dtype=torch.bool, device=dev)  # SGMP: nodes at a fixed face
    for a in range(3):
        for f, at in ((s["fix"][2 * a], ij[a] <= two), (s["fix"][2 * a + 1], ij[a] >= NG[a] - 1 - two)):
            if f == 1:
                fixed |= at
            elif f == 2:
                fixed[a] |= at
            if f:
                bdt[a] |= at
    if sg:  # cells: the 8 nodes, the weights of the centre velocity (mirrored at fixed faces)
        ci = torch.arange(ncell, device=dev)
        cc = (ci % NC[0], ci // NC[0] % NC[1], ci // (NC[0] * NC[1]))
        cnode = [((cc[2] + k) * NG[1] + cc[1] + j) * NG[0] + cc[0] + i for i, j, k in _CORNERS]
        face = torch.zeros(ncell, dtype=torch.bool, device=dev)
        cxx = torch.zeros(3, ncell, dtype=F, device=dev)
        for a in range(3):
            if NC[a] > 1:
                lo, hi = cc[a] == 0, cc[a] == NC[a] - 1
                face |= (lo & (s["fix"][2 * a] != 0)) | (hi & (s["fix"][2 * a + 1] != 0))
                cxx[a] = torch.where(hi, -1.0, torch.where(lo, 1.0, 0.0))
        cxx *= face
        CNC = [max(1, v - 1) for v in NC]

    def scatter(slots, vals, size):
        out = torch.zeros(len(vals), size, dtype=F, device=dev)
        for nd, w, _ in slots():
            out.index_add_(1, nd, torch.stack([u * w for u in vals]))
        return out

    def cells_to_nodes(cv, w=None):
        out = torch.zeros(cv.shape[0], nn, dtype=F, device=dev)
        for k, c in enumerate(cnode):
            out.index_add_(1, c, cv * 0.125 if w is None else w(k))
        return out

    def sg_corner_weights(xx):
        for k, (i, j, l) in enumerate(_CORNERS):
            w = 0.125 * (1 + (2 * i - 1) * xx[0]) * (1 + (2 * j - 1) * xx[1]) * (1 + (2 * l - 1) * xx[2])
            cid = c1 + i + j * NC[0] + l * NC[0] * NC[1]
            ok = cid < ncell
            yield cid.clamp(max=ncell - 1), w * ok, None

    dt, time, istep = h / wave * _f(s["dtsc"]), 0.0, 0
    musl, usf = s["scheme"] == "musl", s["scheme"] == "usf"
    for _ in range(steps):
        istep, time = istep + 1, time + dt
        if sg:
            u = (x - torch.tensor(s0, dtype=F, device=dev)[:, None]) / h
            dc = torch.trunc(u - 0.5).long()
            c1f = (dc[2] * CNC[1] + dc[1]) * CNC[0] + dc[0]
            c1 = ((c1f // (CNC[0] * CNC[1])) * NC[1] + c1f // CNC[0] % CNC[1]) * NC[0] + c1f % CNC[0]
            nd = torch.trunc(u + 0.5).long()
            inode = (nd[2] * NG[1] + nd[1]) * NG[0] + nd[0]
            xi = (u - nd) * 2
            b3 = bdt[:, inode]
            xxn = torch.where(b3, torch.sign(xi), xi)
            xn = (u - torch.floor(u)) * 2 - 1
            xaux = torch.where(b3, torch.where(xn < 0, 1 + 2 * xn, 2 * xn - 1), xxn)
            slots = lambda: sg_corner_weights(xxn)  # noqa: E731
            cm = scatter(slots, [m, m * v[0], m * v[1], m * v[2]], ncell)
            mg, *pg = cells_to_nodes(cm * (cm[0] > cutoff))
            pg = torch.stack(pg)
        else:
            wt = _weights(s["shape"], x, s0, h, NG)
            slots = lambda: _slots(wt, NG)  # noqa: E731
            g = scatter(slots, [m, m * v[0], m * v[1], m * v[2]], nn)
            mg, pg = g[0], g[1:]
        live = mg > cutoff
        im = torch.where(live, 1 / torch.where(live, mg, 1.0), 0.0)

        def stress(vg):
            nonlocal vol, sm, sd, q, H
            L = z(3, 3)
            if sg:
                cf = torch.zeros(9, ncell, dtype=F, device=dev)
                for k, c in enumerate(cnode):
                    for b in range(3):
                        d = (2 * _CORNERS[k][b] - 1) * 0.25 / h
                        for a in range(3):
                            cf[a * 3 + b] += d * vg[a][c]
                for cid, w, _ in slots():
                    L += (cf[:, cid] * w).view(3, 3, -1)
            else:
                for nd_, _, dN in slots():
                    vn = vg[:, nd_]
                    for b in range(3):
                        L[:, b] += vn * dN[b]
            L = L * dt
            de = [L[0, 0], L[1, 1], L[2, 2], L[0, 1] + L[1, 0], L[2, 1] + L[1, 2], L[0, 2] + L[2, 0]]
            w0, w1, w2 = (L[2, 1] - L[1, 2]) / 2, (L[0, 2] - L[2, 0]) / 2, (L[1, 0] - L[0, 1]) / 2
            tr = de[0] + de[1] + de[2]
            vold = vol
            if name == "neoh":
                I3 = torch.eye(3, dtype=F, device=dev)[:, :, None]
                A = L + I3
                det = lambda M: (M[0, 0] * (M[1, 1] * M[2, 2] - M[1, 2] * M[2, 1]) - M[0, 1] * (M[1, 0] * M[2, 2] - M[1, 2] * M[2, 0])  # noqa: E731
                                 + M[0, 2] * (M[1, 0] * M[2, 1] - M[1, 1] * M[2, 0]))
                vol = vold * det(A)
                H = H + L + torch.einsum("ikn,kjn->ijn", L, H)
                Fm = H + I3
                J = det(Fm)
                B = torch.einsum("ikn,jkn->ijn", Fm, Fm) - I3
                p = lam * torch.log(J)
                sig = [(0.5 * G2 * B[0, 0] + p) / J, (0.5 * G2 * B[1, 1] + p) / J, (0.5 * G2 * B[2, 2] + p) / J,
                       0.5 * G2 * B[0, 1] / J, 0.5 * G2 * B[1, 2] / J, 0.5 * G2 * B[0, 2] / J]
                sm = (sig[0] + sig[1] + sig[2]) / 3
                sd = torch.stack([sig[0] - sm, sig[1] - sm, sig[2] - sm, sig[3], sig[4], sig[5]])
            else:
                vol = vold * (1 + tr)
            den = m / vol
            ddot = torch.clamp(tr / dt, max=0.0)  # bulk viscosity acts in compression
            if name == "null":  # weakly compressible: pressure from the density, viscous deviator
                sd = torch.stack([2 * mp[2] * de[0] / dt, 2 * mp[2] * de[1] / dt, 2 * mp[2] * de[2] / dt,
                                  mp[2] * de[3] / dt, mp[2] * de[4] / dt, mp[2] * de[5] / dt])
            elif name != "neoh":
                g = [sd[0] + sm, sd[1] + sm, sd[2] + sm, sd[3], sd[4], sd[5]]
                q1, q2, q3 = 2 * g[3] * w2, 2 * g[5] * w1, 2 * g[4] * w0
                g = [g[0] - q1 + q2, g[1] + q1 - q3, g[2] - q2 + q3,
                     g[3] + w2 * (g[0] - g[1]) + w1 * g[4] - w0 * g[5],
                     g[4] + w0 * (g[1] - g[2]) + w2 * g[5] - w1 * g[3],
                     g[5] + w1 * (g[2] - g[0]) + w0 * g[3] - w2 * g[4]]
                sm = (g[0] + g[1] + g[2]) / 3
                sd = torch.stack([g[0] - sm + G2 * (de[0] - tr / 3), g[1] - sm + G2 * (de[1] - tr / 3), g[2] - sm + G2 * (de[2] - tr / 3),
                                  g[3] + 0.5 * G2 * de[3], g[4] + 0.5 * G2 * de[4], g[5] + 0.5 * G2 * de[5]])
                sm = sm + K3 * tr / 3
                if name == "dpm":
                    qf, kf, qp, ten = mp[3:7]
                    ten = 0.0 if qf == 0 else min(ten, kf / qf)
                    G, K = G2 / 2, K3 / 3
                    tau = torch.sqrt(0.5 * (sd[0] ** 2 + sd[1] ** 2 + sd[2] ** 2) + sd[3] ** 2 + sd[4] ** 2 + sd[5] ** 2)
                    fi = tau + qf * sm - kf
                    ds = sm - ten
                    hf = tau - (kf - qf * ten) - (math.sqrt(1 + qf * qf) - qf) * ds
                    shear = torch.where(ds < 0, fi > 0, hf > 0)
                    smn = sm - K * qp * fi / (G + K * qf * qp)
                    ratio = torch.where(shear, (kf - qf * smn) / torch.where(shear, tau, 1.0), 1.0)
                    sm = torch.where(shear, smn, torch.where(ds < 0, sm, ten))
                    sd = sd * ratio
            # (the null material decides on its pressure before the step's)
            q = torch.where(sm < 0, den * h * h * s["bq"][0] * ddot ** 2 - s["bq"][1] * den * h * cp0 * ddot, 0.0)
            if name == "null":
                sm = -c0 * c0 * (den - rho)

        if usf:
            pg = torch.where(fixed, 0.0, pg)
            stress(pg * im)
        fext = fxp * (time / _f(s["qload"]) if s["qload"] and time < _f(s["qload"]) else 1.0)
        if s["damp"]:
            fext = fext - _f(s["damp"]) * m * v
        fext = fext + m * grav
        p = sm - q
        sv = [(sd[0] + p) * vol, (sd[1] + p) * vol, (sd[2] + p) * vol, sd[3] * vol, sd[4] * vol, sd[5] * vol]
        if sg:
            cf = scatter(slots, [fext[0], fext[1], fext[2]] + sv, ncell)

            def corner_force(k):
                d = [(2 * _CORNERS[k][b] - 1) * 0.25 / h for b in range(3)]
                return torch.stack([0.125 * cf[0] - (cf[3] * d[0] + cf[6] * d[1] + cf[8] * d[2]),
                                    0.125 * cf[1] - (cf[6] * d[0] + cf[4] * d[1] + cf[7] * d[2]),
                                    0.125 * cf[2] - (cf[8] * d[0] + cf[7] * d[1] + cf[5] * d[2])])
            fg = cells_to_nodes(cf[:3], corner_force)
        else:
            fg = torch.zeros(3, nn, dtype=F, device=dev)
            for nd_, w, d in slots():
                fg.index_add_(1, nd_, torch.stack([fext[0] * w - (sv[0] * d[0] + sv[3] * d[1] + sv[5] * d[2]),
                                                   fext[1] * w - (sv[3] * d[0] + sv[1] * d[1] + sv[4] * d[2]),
                                                   fext[2] * w - (sv[5] * d[0] + sv[4] * d[1] + sv[2] * d[2])]))
        pg = pg + fg * (dt * (0.5 if istep == 1 else 1.0))
        pg, fg = torch.where(fixed, 0.0, pg), torch.where(fixed, 0.0, fg)
        vg, ag = pg * im, fg * im
        vp, ap = z(3), z(3)
        if sg:
            cv = torch.zeros(6, ncell, dtype=F, device=dev)
            for k, c in enumerate(cnode):
                w = 0.125
                for b in range(3):
                    w = w * (1 + (2 * _CORNERS[k][b] - 1) * cxx[b])
                cv += torch.cat([vg[:, c], ag[:, c]]) * w
            for cid, w, _ in sg_corner_weights(xaux):
                vp += cv[:3, cid] * w
                ap += cv[3:, cid] * w
        else:
            for nd_, w, _ in slots():
                vp += vg[:, nd_] * w
                ap += ag[:, nd_] * w
        xnew = x + vp * dt
        v = v + ap * (dt * (0.5 if istep == 1 else 1.0))
        if musl:
            mv = [m * v[0], m * v[1], m * v[2]]
            pg = cells_to_nodes(scatter(slots, mv, ncell)) if sg else scatter(slots, mv, nn)
            pg = torch.where(fixed, 0.0, pg)
            vg = pg * im
        if not usf:
            stress(vg)
        x = xnew
        dt = h / (wave + float(v.abs().max())) * _f(s["dtsc"])
    return {"Xp": x, "VXp": v, "SM": sm, "SD": sd}
