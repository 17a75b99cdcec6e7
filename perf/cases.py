"""The work a user of godar_b200 has it do, as measurable cases.

A case is a dict of plain values.  Five kinds:

``step``   one floe field on the GPU (``Stepper``), advanced by ``steps`` time
           steps and read back.  ``call`` "block": one call for all steps, the
           state read back.  ``call`` "queued": one queued call per time step,
           the way the Fortran driver calls its stepper, the last one with
           diagnostics, then the whole output step (every per-floe output, the
           contact list and the bond list).
``batch``  many fields in one ``Batch`` (an ensemble), advanced together, then
           positions and velocities of every floe read back.  ``monitor``: a
           forcing upload and a per-field summary at every step.
``serve``  one turn of the request loop: a field joins the resident ones, all
           advance by a chunk of steps, the field is read and leaves.
``cold``   a field from its host arrays to its first step and back: context,
           upload, bond creation, neighbour search, one step, read-back.
``place``  an initial field of non-overlapping disks.

Steps that are timed come after the batch has run its first 20 (18 of them
choose launch configurations): a run takes thousands.
"""
import math
import os
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from godar_b200 import generators as gen
from godar_b200 import lib as gl
from godar_b200.params import (BC_OPEN_BOTTOM, BC_OPEN_LEFT, BC_OPEN_RIGHT, BC_OPEN_TOP, BC_PERIODIC_X,
                               BC_PERIODIC_Y, PREC_FP64, PREC_MIXED)

WARM = 20
PREC = {"fp64": PREC_FP64, "mixed": PREC_MIXED}
STATE = ["x", "y", "u", "v", "r", "h", "theta", "omega"]


def listed():
    return [
        # the smallest field (configuration 1: 256 disks between four walls), stepped as the Fortran driver does,
        # with its output step: launches and latency
        {"name": "lattice256_walls_fp64", "kind": "step", "field": "lattice", "n": 256, "periodic": False,
         "precision": "fp64", "steps": 32, "call": "queued"},
        # configuration 1, doubly periodic, in mixed precision, one call for many steps
        {"name": "lattice256_mixed", "kind": "step", "field": "lattice", "n": 256, "periodic": True,
         "precision": "mixed", "steps": 64, "call": "block"},
        # a small bonded field of no round size
        {"name": "bonded1021_fp64", "kind": "step", "field": "bonded", "n": 1021, "precision": "fp64",
         "steps": 64, "call": "block"},
        # configuration 2 (4,096 bonded floes under a wind field), stepped by the driver, plain precision
        {"name": "bonded4096_fp64", "kind": "step", "field": "bonded", "n": 4096, "precision": "fp64",
         "steps": 32, "call": "queued"},
        # configuration 2 in mixed precision
        {"name": "bonded4096_mixed", "kind": "step", "field": "bonded", "n": 4096, "precision": "mixed",
         "steps": 64, "call": "block"},
        # configuration 3's kind (65,536 floes, sheltering, ridging, a wall, gridded forcing): every candidate pair acts
        {"name": "poly65536_fp64", "kind": "step", "field": "poly", "n": 65536, "precision": "fp64",
         "steps": 8, "call": "block"},
        {"name": "poly65536_mixed", "kind": "step", "field": "poly", "n": 65536, "precision": "mixed",
         "steps": 8, "call": "queued"},
        # configuration 4: the 512-field ensemble (2.2 M floes), its forcing and a summary at every step
        {"name": "ensemble512_mixed", "kind": "batch", "count": 512, "lo": 256, "hi": 16384, "precision": "mixed",
         "steps": 16, "monitor": True},
        # the plain method over a quarter of it
        {"name": "ensemble128_fp64", "kind": "batch", "count": 128, "lo": 256, "hi": 16384, "precision": "fp64",
         "steps": 16, "monitor": False},
        # configuration 5: a request of the served stream joins six others
        {"name": "serve_mixed", "kind": "serve", "residents": 6, "lo": 512, "hi": 65536, "n": 5793,
         "precision": "mixed", "steps": 50},
        # a new field's first step
        {"name": "cold4096_fp64", "kind": "cold", "field": "bonded", "n": 4096, "precision": "fp64"},
        # an initial field
        {"name": "place32768", "kind": "place", "n": 32768, "phi": 0.66},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 10 + ["batch"] * 4 + ["serve"] * 2 + ["cold"] * 2 + ["place"] * 2)
    prec = rng.choice(["fp64", "mixed"])
    if kind == "step":
        field = rng.choice(["bonded", "bonded", "lattice", "poly"])
        c = {"kind": kind, "field": field, "precision": prec, "call": rng.choice(["block", "queued"])}
        if field == "lattice":
            c.update(n=rng.randint(7, 16) ** 2, periodic=rng.random() < 0.5, steps=rng.randint(16, 64))
        elif field == "bonded":
            c.update(n=_log_int(rng, 64, 32768), steps=rng.randint(16, 64))
        else:
            c.update(n=_log_int(rng, 512, 65536), steps=rng.randint(4, 8))
        return c
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 2, 128 if prec == "fp64" else 512), "lo": 256,
                "hi": rng.choice([1024, 4096, 16384]), "precision": prec, "steps": rng.randint(6, 16),
                "monitor": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "residents": rng.randint(1, 8), "lo": 512, "hi": rng.choice([8192, 65536]),
                "n": _log_int(rng, 512, 16384), "precision": prec, "steps": rng.randint(10, 50)}
    if kind == "cold":
        return {"kind": kind, "field": rng.choice(["bonded", "bonded", "poly"]), "n": _log_int(rng, 512, 16384),
                "precision": prec}
    return {"kind": kind, "n": _log_int(rng, 512, 32768), "phi": round(rng.uniform(0.55, 0.66), 3)}


# ------------------------------------------------------------------ inputs
def _field(case, seed):
    if case["field"] == "lattice":
        f = gen.lattice_field(math.isqrt(case["n"]), case["periodic"], seed=seed)
        # at the configuration's 1 s the stiff contacts of a field pressed against its walls blow up in the end
        f.params.dt = 0.2
        return f
    if case["field"] == "bonded":
        return gen.bonded_field(case["n"], seed=seed)
    return _poly(case["n"], seed)


def _poly(n, seed):
    """Configuration 3's field (polydisperse_field: r^-2 radii, gamma thickness, a wall, sheltering, ridging, gridded
    wind and current, a tenth of the close pairs bonded) with radii of [400, 2000] m, no floe thinner than 0.3 m and
    75 % area fraction: over the thousands of steps of a measurement some draws of [100, 5000] m blow up, when a
    contact of a small with a large floe begins within the rounding of its chord."""
    f = gen.polydisperse_field(512, seed=seed, dt=0.01)
    rng = np.random.default_rng(seed)
    a, b = 400.0, 2000.0
    r = 1.0 / (1.0 / a - rng.uniform(0.0, 1.0, n) * (1.0 / a - 1.0 / b))
    h = np.maximum(rng.gamma(2.0, 0.75, n), 0.3)
    x, y, Lx, Ly, _ = gen.place_fraction(r, 0.75, 1.0, False, True, seed, 200)
    f.params.nx, f.params.ny = Lx, Ly
    return gen.Field("poly", f.params, x, y, r, h, 2000, forcing=f.forcing)


def _member(n, seed, phi):
    rng = np.random.default_rng(seed)
    return gen.bonded_field(n, seed=seed, phi=phi, wind_field=False, wind_dir_deg=rng.uniform(0.0, 360.0),
                            wind_speed=rng.uniform(8.0, 16.0), max_trials=200)


def _sizes(case, count):
    """The sizes of a batch's fields follow from the case alone."""
    rng = random.Random(1000003 * count + 31 * case["hi"] + case["lo"])
    return [_log_int(rng, case["lo"], case["hi"]) for _ in range(count)]


def _members(sizes, seed, phi):
    jobs = sorted(range(len(sizes)), key=lambda k: -sizes[k])
    with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
        done = dict(zip(jobs, ex.map(lambda k: _member(sizes[k], 100003 * (seed + 1) + k, phi), jobs)))
    return [done[k] for k in range(len(sizes))]


def _stepper(f, precision):
    s = gl.Stepper(f.params, f.n, PREC[precision])
    s.upload(f.x, f.y, f.r, f.h, f.theta, f.omega, f.u, f.v, f.bonds, f.damage)
    if f.forcing is not None:
        s.set_field(f.forcing)
    return s


def _radii(case, seed):
    rng = np.random.default_rng(seed)
    r = np.clip(rng.lognormal(math.log(800.0), 0.4, case["n"]), 200.0, 3000.0)
    return r, math.sqrt(float(np.sum(np.pi * r * r)) / case["phi"])


def _fields(case, seed):
    """The fields of a batch or of a request loop (the arriving one last)."""
    if case["kind"] == "batch":
        return _members(_sizes(case, case["count"]), seed, 0.74)
    return _members(_sizes(case, case["residents"]) + [case["n"]], seed, 0.70)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        f = _field(case, seed)
        s = _stepper(f, case["precision"])
        s.set_diagnostics(False)
        s.step(1, 0, WARM)
        return {"case": case, "s": s, "t": WARM}
    if kind == "cold":
        return {"case": case, "f": _field(case, seed)}
    if kind == "place":
        r, side = _radii(case, seed)
        return {"case": case, "r": r, "side": side, "seed": seed}
    fields = _fields(case, seed)
    b = gl.Batch(PREC[case["precision"]])
    b.set_diagnostics(False)
    new = fields.pop() if kind == "serve" else None
    for f in fields:
        b.add_field(f)
    b.step(WARM)
    st = {"case": case, "b": b, "f": new}
    if kind == "batch":
        _, n = b.count()
        st["out"] = [torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
        st["sum"] = [torch.empty(4 * len(fields), dtype=torch.float64, pin_memory=True).numpy() for _ in range(2)]
        st["uvw"] = np.array([[f.params.ua, f.params.va, f.params.uw, f.params.vw] for f in fields])
    return st


# ------------------------------------------------------------------ the calls
def _padded(n, i, j, val):
    """A pair list in arrays of one length for a field of n floes."""
    full = [np.full(8 * n, -1, np.int32), np.full(8 * n, -1, np.int32), np.zeros(8 * n)]
    for a, b in zip(full, (i, j, val)):
        if b is not None:
            a[:len(b)] = b
    return full


def _pairs_out(out, name, lists):
    for part, a in zip(("i", "j", "value"), lists):
        out[f"{name}_{part}"] = a


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        s, t, k = st["s"], st["t"], case["steps"]
        st["t"] = t + k
        if case["call"] == "block":
            s.step(t + 1, 0, k)
            return s.floes(STATE)
        for q in range(1, k):
            s.step_async(t + q)
        s.set_diagnostics(True)
        s.step_async(t + k)
        s.set_diagnostics(False)
        out, contacts = s.download(which=gl.P_CONTACTS)
        _pairs_out(out, "contact", _padded(case["n"], *contacts))
        _pairs_out(out, "bond", _padded(case["n"], *s.pairs(gl.P_BONDS)))
        return out
    if kind == "batch":
        b = st["b"]
        if case["monitor"]:
            for q in range(case["steps"]):
                b.set_uniform_forcing(st["uvw"])
                b.step_async(1)
                b.summary_async(st["sum"][q & 1])
        else:
            b.step(case["steps"])
        b.get_all_async(["x", "y", "u", "v"], st["out"])
        b.wait()
        return st["out"]
    if kind == "serve":
        b = st["b"]
        hid = b.add_field(st["f"])
        b.step(case["steps"])
        out = [b.field(hid, k) for k in ("x", "y", "u", "v")]
        b.remove(hid)
        return out
    if kind == "cold":
        f = st["f"]
        s = _stepper(f, case["precision"])
        s.step(1, 0, 1)
        out, bonds = s.download(which=gl.P_BONDS)
        s.close()
        _pairs_out(out, "bond", _padded(case["n"], *bonds))
        return out
    x, y, placed = gl.place_disks(st["r"], st["side"], st["side"], True, True, st["seed"])
    return [x, y, placed]


# ------------------------------------------------------------------ bytes and operations
# Per floe: bonds, and pairs close enough to need a test at a step, in these fields.
BONDS = {"lattice": 0.0, "bonded": 1.55, "poly": 0.3}
PAIRS = {"lattice": 1.0, "bonded": 1.5, "poly": 16.0}


def work(case):
    kind = case["kind"]
    if kind == "place":
        n = case["n"]
        # radii in, positions out; a few hundred distance tests a disk
        return {"bytes": 24.0 * n, "flops": 400.0 * 8 * n}
    if kind == "cold":
        n, field = case["n"], case["field"]
        steps, read = 1, 22
    elif kind == "step":
        n, field = case["n"], case["field"]
        steps, read = case["steps"], 22 if case["call"] == "queued" else 8
    else:
        sizes = _sizes(case, case["count"] if kind == "batch" else case["residents"])
        n, field = sum(sizes) + (case["n"] if kind == "serve" else 0), "bonded"
        steps, read = case["steps"], 4
    nb, npair = BONDS[field] * n, PAIRS[field] * n
    # a step reads and writes the eight state values of a floe, the five of a bond's strain and damage (and reads its
    # three of geometry) and the history of a pair in contact (about one floe in sixteen); a field that stays
    # on the chip from step to step need only do so once
    state = 128.0 * n + 104.0 * nb + 64.0 * n / 16
    moved = state * (steps if state > 126e6 else 1) + 8.0 * read * n
    return {"bytes": moved, "flops": steps * (150.0 * n + 250.0 * nb + 15.0 * npair)}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "place":
        return None
    if kind == "step":
        f, steps = _field(case, seed), WARM + case["steps"]
    elif kind == "cold":
        f, steps = _field(case, seed), 1
    else:
        sizes = _sizes(case, case["count"]) if kind == "batch" else [case["n"]]
        steps = case["steps"] + (WARM if kind == "batch" else 0)
        if sum(sizes) * steps > 5.5e6:
            return None
        outs = []
        for f in (_fields(case, seed) if kind == "batch" else _fields(case, seed)[-1:]):
            sim = _Sim(f)
            for q in range(steps):
                sim.step(False)
            outs.append([sim.s[k] for k in ("x", "y", "u", "v")])
        return [np.concatenate([o[k] for o in outs]) for k in range(4)]
    if f.n * PAIRS[case["field"]] * steps > 6e7:
        return None
    sim = _Sim(f)
    for q in range(steps):
        sim.step(q == steps - 1)
    if kind == "step" and case["call"] == "block":
        return {k: sim.s[k] for k in STATE}
    out = {k: sim.s[k] for k in STATE}
    out.update(sim.diag)
    if kind == "step":
        _pairs_out(out, "contact", [None, None, _padded(f.n, None, None, sim.overlaps)[2]])
    _pairs_out(out, "bond", [None, None, _padded(f.n, None, None, sim.bonds())[2]])
    return out


class _Sim:
    """The time step of the reference (model/src/stepper.f90:44-343 and the routines it calls) in 64-bit numpy,
    whole arrays at a time."""

    def __init__(self, f):
        self.p = p = f.params
        n = f.n
        z = lambda a: np.zeros(n) if a is None else np.array(a, dtype=np.float64)  # noqa: E731
        self.s = {"x": z(f.x), "y": z(f.y), "u": z(f.u), "v": z(f.v), "r": z(f.r), "h": z(f.h), "theta": z(f.theta),
                  "omega": z(f.omega)}
        self.n = n
        self.grid = None if f.forcing is None else np.asarray(f.forcing, np.float64).reshape(4, p.field_ny, p.field_nx)
        self.px, self.py = bool(p.boundary & BC_PERIODIC_X), bool(p.boundary & BC_PERIODIC_Y)
        self.wall = {k: np.zeros(n) for k in ("t1", "t2", "th1", "th2")}
        # every pair that can come within the search radius while no floe moves further than half of this
        self.skin = 0.03 * (float(self.s["r"].max()) + p.rtree)
        self.x0, self.y0 = self.s["x"].copy(), self.s["y"].copy()
        self.i, self.j = self._pairs(float(self.s["r"].max()) + p.rtree + self.skin)
        m = len(self.i)
        self.hist = {k: np.zeros(m) for k in ("t", "th", "fcn", "fct")}
        self._make_bonds()

    def _off(self, a, b, L, per):
        d = a - b
        if per:
            d = np.where(d > 0.5 * L, d - L, np.where(d < -0.5 * L, d + L, d))
        return d

    def _pairs(self, R):
        """i < j with dist <= r_i + rtree + skin, by a cell list."""
        p, x, y, r = self.p, self.s["x"], self.s["y"], self.s["r"]
        lo_x, lo_y = (0.0 if self.px else x.min()), (0.0 if self.py else y.min())
        Lx = p.nx if self.px else max(x.max() - lo_x, 1.0)
        Ly = p.ny if self.py else max(y.max() - lo_y, 1.0)
        ncx, ncy = max(1, int(Lx // R)), max(1, int(Ly // R))
        cx = np.clip(((x - lo_x) / Lx * ncx).astype(np.int64), 0, ncx - 1)
        cy = np.clip(((y - lo_y) / Ly * ncy).astype(np.int64), 0, ncy - 1)
        cell = cy * ncx + cx
        order = np.argsort(cell, kind="stable")
        start = np.searchsorted(cell[order], np.arange(ncx * ncy + 1))
        found = []
        seen = set()
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                ax, ay = cx + ox, cy + oy
                key = (ox % ncx if self.px else ox, oy % ncy if self.py else oy)
                if key in seen:
                    continue
                seen.add(key)
                ok = np.ones(self.n, bool)
                if self.px:
                    ax = ax % ncx
                else:
                    ok &= (ax >= 0) & (ax < ncx)
                if self.py:
                    ay = ay % ncy
                else:
                    ok &= (ay >= 0) & (ay < ncy)
                a = np.nonzero(ok)[0]
                c = ay[a] * ncx + ax[a]
                cnt = start[c + 1] - start[c]
                i = np.repeat(a, cnt)
                at = np.arange(cnt.sum()) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(start[c], cnt)
                j = order[at]
                keep = i < j
                i, j = i[keep], j[keep]
                dx, dy = self._off(x[i], x[j], p.nx, self.px), self._off(y[i], y[j], p.ny, self.py)
                keep = np.sqrt(dx * dx + dy * dy) <= r[i] + p.rtree + self.skin
                found.append((i[keep], j[keep]))
        i, j = (np.concatenate([q[k] for q in found]) for k in (0, 1))
        o = np.lexsort((j, i))
        return i[o], j[o]

    def _make_bonds(self):
        p, s = self.p, self.s
        m = len(self.i)
        self.bond = np.zeros(m, bool)
        names = ("rb", "hb", "lb", "sb", "ib", "dnb", "dtb", "thji", "thij", "dmg")
        self.b = {k: np.zeros(m) for k in names}
        if not p.cohesion:
            return
        i, j = self.i, self.j
        dx, dy = self._off(s["x"][i], s["x"][j], p.nx, self.px), self._off(s["y"][i], s["y"][j], p.ny, self.py)
        d = np.sqrt(dx * dx + dy * dy)
        ri, rj = s["r"][i], s["r"][j]
        sel = (d <= ri + p.rtree) & ((ri + rj) - d >= -(p.bond_lim + p.bond_lim_rel * (ri + rj)))
        if 0.0 < p.bond_frac < 1.0:
            u32 = np.uint32
            with np.errstate(over="ignore"):
                h = (u32(p.bond_seed) * u32(0x9e3779b9)) ^ (i.astype(u32) * u32(0x85ebca6b)) \
                    ^ (j.astype(u32) * u32(0xc2b2ae35) + u32(0x27d4eb2f))
                h ^= h >> u32(16)
                h *= u32(0x7feb352d)
                h ^= h >> u32(15)
                h *= u32(0x846ca68b)
                h ^= h >> u32(16)
            sel &= h.astype(np.float64) * 2.0 ** -32 < p.bond_frac
        self.bond = sel
        self.has_bond = sel.copy()
        B = self.b
        B["rb"] = p.lambda_rb * np.minimum(ri, rj)
        B["hb"] = (s["h"][i] + s["h"][j]) / 2.0
        B["lb"] = d
        B["sb"] = 2.0 * B["rb"] * B["hb"]
        B["ib"] = 2.0 / 3.0 * B["hb"] * B["rb"] ** 3

    def bonds(self):
        """Damage of the live bonds, by (i, j)."""
        return self.b["dmg"][self.bond]

    def _wind(self):
        p, s = self.p, self.s
        if self.grid is None:
            return tuple(np.full(self.n, v) for v in (p.ua, p.va, p.uw, p.vw))
        fnx, fny = p.field_nx, p.field_ny
        fx = np.clip(s["x"], 0.0, p.nx) / p.nx * (fnx - 1)
        fy = np.clip(s["y"], 0.0, p.ny) / p.ny * (fny - 1)
        ix = np.minimum(np.floor(fx).astype(np.int64), fnx - 2)
        iy = np.minimum(np.floor(fy).astype(np.int64), fny - 2)
        tx, ty = fx - ix, fy - iy
        F = self.grid
        g = [(1 - ty) * ((1 - tx) * F[c, iy, ix] + tx * F[c, iy, ix + 1])
             + ty * ((1 - tx) * F[c, iy + 1, ix] + tx * F[c, iy + 1, ix + 1]) for c in range(4)]
        return p.ua + g[0], p.va + g[1], p.uw + g[2], p.vw + g[3]

    @staticmethod
    def _fit(xi):
        return (0.9117 * xi * xi + 0.2722 * xi + 0.003324) / (xi * xi + 1.524 * xi + 0.03159)

    @staticmethod
    def _heavi(x):
        return np.copysign(0.5, x) + 0.5

    def _shelter(self, hfi, hfj, dn, c, s, u, v):
        wn = np.sqrt(u * u + v * v) + 1e-20
        ct = (u * c + v * s) / wn
        ex = np.exp(-(float(np.float32(0.18)) * np.abs(dn / ct)) / hfj)
        hd = self._heavi(dn)
        D = (1 - (1 - hd) * (1 - ex)) - hd * self._heavi(hfi - hfj) * (1 - hfj / hfi)
        return 1 - D * self._heavi(ct) * ct

    def _props(self, r, h):
        p = self.p
        mass = p.rhoice * p.pi * h * r * r
        return mass, 0.5 * mass * r * r

    def _grow(self, r, h, vol):
        dh = vol / (self.p.pi * r * r)
        return r * np.sqrt(h / (h + dh)), h + dh

    def step(self, diag):
        with np.errstate(all="ignore"):
            self._step(diag)

    def _step(self, diag):
        p, S, n = self.p, self.s, self.n
        dt = p.dt
        x, y, u, v, om, r, h = (S[k] for k in ("x", "y", "u", "v", "omega", "r", "h"))
        moved = np.hypot(self._off(x, self.x0, p.nx, self.px), self._off(y, self.y0, p.ny, self.py)).max()
        if moved > 0.5 * self.skin:
            raise RuntimeError("a floe has left its neighbour list")
        mass, inert = self._props(r, h)
        wind = self._wind()
        add = lambda idx, w: np.bincount(idx, weights=w, minlength=n)  # noqa: E731
        i0, j0 = self.i, self.j
        dx0, dy0 = self._off(x[i0], x[j0], p.nx, self.px), self._off(y[i0], y[j0], p.ny, self.py)
        d0 = np.sqrt(dx0 * dx0 + dy0 * dy0)
        cand = np.nonzero(d0 <= r[i0] + p.rtree)[0]
        H, B = self.hist, self.b
        dn0 = (r[i0] + r[j0]) - d0
        acc = {k: np.zeros(n) for k in ("fcx", "fcy", "mc", "fbx", "fby", "mb", "tac", "pc", "tab", "pb", "sxx", "syy",
                                        "sxy", "syx")}
        ri_all, rj_all = r[i0], r[j0]
        hi_all, hj_all = h[i0], h[j0]

        def frame(k):
            i, j, d = i0[k], j0[k], d0[k]
            c, s = -dx0[k] / d, -dy0[k] / d
            du, dv = u[j] - u[i], v[j] - v[i]
            return i, j, d, c, s, du * c + dv * s, -(du * s) + dv * c

        # ---- contacts
        touch = cand[dn0[cand] > 0.0]
        away = cand[dn0[cand] <= 0.0]
        H["t"][away] = 0.0
        H["th"][away] = 0.0
        events = []
        if len(touch):
            k = touch
            i, j, d, c, s, veln, vb = frame(k)
            ri, rj, hi, hj, dn = r[i], r[j], h[i], h[j], dn0[k]
            velt = vb - (om[i] * ri + om[j] * rj)
            omr = om[j] - om[i]
            dtan = H["t"][k] - velt * dt
            thr = H["th"][k] - omr * dt

            def chord(ri, rj):
                q = (d * d - rj * rj + ri * ri) / (2 * d)
                return 2 * np.sqrt(ri * ri - q * q)
            dr = chord(ri, rj)
            mred, rred, hmin = mass[i] * mass[j] / (mass[i] + mass[j]), ri * rj / (ri + rj), np.minimum(hi, hj)
            knc = p.pi * p.ec * hmin * self._fit(dn * rred / (2 * hmin * hmin))
            kn = knc
            ratio = 6 * p.gc / p.ec

            def damp(kn, dr):
                ktc = ratio * kn
                gn = -(p.beta * np.sqrt(4 * kn * mred))
                return (ktc, kn * dr * dr / 12, gn, -(2 * p.beta * np.sqrt(2.0 / 3.0 * ktc * mred)), gn * dr * dr / 12)
            ktc, krc, gn, gt, gr = damp(kn, dr)
            fcn = np.maximum(knc * dn - gn * veln, 0.0)
            ri_l, rj_l, hi_l, hj_l = ri.copy(), rj.copy(), hi.copy(), hj.copy()
            if p.ridging:
                pl = p.sigmanc_crit * hmin <= fcn / dr / hmin
                if pl.any():
                    knp = p.sigmanc_crit * hmin * hmin * dr / dn
                    two = damp(knp, dr)
                    ktc, krc, gn, gt, gr = (np.where(pl, b, a) for a, b in zip((ktc, krc, gn, gt, gr), two))
                    fcn = np.where(pl, np.minimum(fcn, p.sigmanc_crit * hmin * hmin * dr), fcn)
                    dij, dji = (d * d - rj * rj + ri * ri) / (2 * d), (d * d - ri * ri + rj * rj) / (2 * d)
                    area = ri * ri * np.arccos(dij / ri) - dij * dr / 2 + rj * rj * np.arccos(dji / rj) - dji * dr / 2
                    vol = np.maximum(area * hmin / 2, 0.0)
                    one = pl & (hmin == hi)
                    two = pl & ~one & (hmin == hj)
                    a, b = self._grow(ri, hi, vol)
                    ri_l, hi_l = np.where(one, a, ri), np.where(one, b, hi)
                    a, b = self._grow(rj, hj, vol)
                    rj_l, hj_l = np.where(two, a, rj), np.where(two, b, hj)
                    dr = np.where(pl, chord(ri_l, rj_l), dr)
                    for q in np.nonzero(one)[0]:
                        events.append((i[q], 1, d[q], vol[q]))
                    for q in np.nonzero(two)[0]:
                        events.append((j[q], 0, i[q], vol[q]))
            fct = ktc * dtan - gt * velt
            slip = np.abs(fct) > p.friction_coeff * np.abs(fcn)
            fct = np.where(slip, -(p.friction_coeff * np.abs(fcn) * np.copysign(1.0, velt)), fct)
            if p.slipping:
                dtan = np.where(slip, (fct + gt * velt) / ktc, dtan)
            mcc = np.where(self.bond[k] | (np.abs(thr) > 2 * np.abs(fcn) / knc / dr), 0.0, krc * thr - gr * omr)
            H["t"][k], H["th"][k], H["fcn"][k], H["fct"][k] = dtan, thr, fcn, fct
            fx, fy = -fcn * c + fct * s, -fcn * s - fct * c
            acc["fcx"] += add(i, fx) - add(j, fx)
            acc["fcy"] += add(i, fy) - add(j, fy)
            acc["mc"] += add(i, -ri_l * fct - mcc) + add(j, -rj_l * fct + mcc)
            ac = dr * np.minimum(hi_l, hj_l)
            acc["tac"] += add(i, ac) + add(j, ac)
            acc["pc"] -= add(i, fcn * ac) + add(j, fcn * ac)
            ri_all[k], rj_all[k] = ri_l, rj_l
            hi_all[k], hj_all[k] = hi_l, hj_l

        # ---- bonds
        stress = np.zeros(len(i0))
        k = cand[self.bond[cand]]
        if len(k):
            i, j, d, c, s, veln, vb = frame(k)
            B["dnb"][k] += veln * dt
            B["dtb"][k] += vb * dt
            B["thji"][k] += om[i] * dt
            B["thij"][k] += om[j] * dt
            dnb, dtb, tj, ti = B["dnb"][k], B["dtb"][k], B["thji"][k], B["thij"][k]
            mi, Ii = self._props(ri_all[k], hi_all[k])
            mj, Ij = self._props(rj_all[k], hj_all[k])
            mred, ired = mi * mj / (mi + mj), Ii * Ij / (Ii + Ij)
            L, sb, ib, rb, hb, D = (B[q][k] for q in ("lb", "sb", "ib", "rb", "hb", "dmg"))
            EA, EI = (1 - D) * p.eb * sb, (1 - D) * p.eb * ib
            ei, ea = 2 * np.sqrt(EI * ired / L), 2 * np.sqrt(EA * mred * L)
            s2, g2 = 6 * EI / L ** 2, 6 * ei / L ** 2
            r1, r2, q1, q2 = 4 * EI / L, 2 * EI / L, 4 * ei / L, 2 * ei / L
            fbn = EA / L * dnb + ea / L * veln
            fbt = 12 * EI / L ** 3 * dtb + s2 * (tj + ti) + 12 * ei / L ** 3 * vb + g2 * (om[i] + om[j])
            mji = r1 * tj + r2 * ti - s2 * dtb + q1 * om[i] + q2 * om[j] - g2 * vb
            mij = r2 * tj + r1 * ti - s2 * dtb + q2 * om[i] + q1 * om[j] - g2 * vb
            st, sc = -fbn / sb + np.abs(mji) * rb / ib, fbn / sb + np.abs(mji) * rb / ib
            phi = (np.abs(fbt) / sb / (p.tau_crit * hb)) ** 2
            phi = phi + np.where(sc > 0, (sc / (p.sigmacb_crit * hb)) ** 2, 0.0)
            phi = phi + np.where(st > 0, (st / (p.sigmatb_crit * hb)) ** 2, 0.0)
            psi = np.minimum(1.0, 1 / np.sqrt(phi))
            D = D + (1 - psi) * (1 - D) * dt / p.dtd - D * dt / p.dth
            broke = D >= p.dmax
            B["dmg"][k] = np.where(broke, 1.0, D)
            self.bond[k[broke]] = False
            fbn, fbt, mji, mij = (np.where(broke, 0.0, a) for a in (fbn, fbt, mji, mij))
            sb = np.where(broke, 0.0, sb)
            fx, fy = fbn * c - fbt * s, fbn * s + fbt * c
            acc["fbx"] += add(i, fx) - add(j, fx)
            acc["fby"] += add(i, fy) - add(j, fy)
            acc["mb"] += add(i, -p.lambda_lb * ri_all[k] * fbt - mji) + add(j, -p.lambda_lb * rj_all[k] * fbt - mij)
            acc["tab"] += add(i, sb) + add(j, sb)
            acc["pb"] -= add(i, fbn * sb) + add(j, fbn * sb)
            stress[k] = np.sqrt(fbn * fbn + fbt * fbt)

        # ---- sheltering and the stress sums: every candidate
        ha = (p.rhowater - p.rhoice) / p.rhowater
        hw = p.rhoice / p.rhowater
        sca = np.ones(n) if p.shelter else np.zeros(n)
        scw = sca.copy()
        if p.shelter or diag:
            i, j, d, c, s, _, _ = frame(cand)
            if p.shelter:
                ua, va, uw, vw = (w[i] for w in wind)
                dn, hi, hj = dn0[cand], hi_all[cand], hj_all[cand]
                hai, haj, hwi, hwj = ha * hi, ha * hj, hw * hi, hw * hj

                def part(a):
                    # four factors of a piece of the pairs that stays in the cache
                    q = slice(a, a + 32768)
                    with np.errstate(all="ignore"):
                        return [self._shelter(f1[q], f2[q], dn[q], g * c[q], g * s[q], wu[q], wv[q])
                                for f1, f2, g, wu, wv in ((hai, haj, 1.0, ua, va), (hwi, hwj, 1.0, uw, vw),
                                                          (haj, hai, -1.0, ua, va), (hwj, hwi, -1.0, uw, vw))]
                with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
                    got = list(ex.map(part, range(0, len(i), 32768)))
                for k4, (least, at) in enumerate(((sca, j), (scw, j), (sca, i), (scw, i))):
                    if got:
                        np.minimum.at(least, at, np.concatenate([g[k4] for g in got]))
            if diag:
                q = (np.sqrt(H["fcn"][cand] ** 2 + H["fct"][cand] ** 2) + stress[cand]) * ri_all[cand]
                for name, a, b in (("sxx", c, c), ("syy", s, s), ("sxy", s, c), ("syx", c, s)):
                    acc[name] -= add(i, q * a * b) + add(j, q * a * b)
        if diag:
            self.overlaps = dn0[touch]     # by (i, j)

        # ---- ridging events of each floe in the order of its sums
        r1, h1 = r.copy(), h.copy()
        for fl, own, _, vol in sorted(events, key=lambda e: e[:3]):
            r1[fl], h1[fl] = self._grow(r1[fl], h1[fl], vol)

        # ---- walls
        W = {q: np.zeros(n) for q in ("fx", "fy", "m", "sxx", "syy", "sxy", "syx", "ta", "p")}
        b = p.boundary
        t1, t2 = np.zeros(n, bool), np.zeros(n, bool)
        for solid, horizontal, far, hit in (
                (not self.py and not b & BC_OPEN_BOTTOM, 0, 0, t1), (not self.py and not b & BC_OPEN_TOP, 0, 1, t1),
                (not self.px and not b & BC_OPEN_LEFT, 1, 0, t2), (not self.px and not b & BC_OPEN_RIGHT, 1, 1, t2)):
            if not solid:
                continue
            pos, edge = (x, p.nx) if horizontal else (y, p.ny)
            k = np.nonzero((pos + r1 > edge) if far else (pos - r1 < 0.0))[0]
            if len(k):
                hit[k] = True
                self._walls(k, horizontal, far, pos, edge, r1, h1, W)
        for hit, a, c in ((t1, "t1", "th1"), (t2, "t2", "th2")):
            self.wall[a][~hit] = 0.0
            self.wall[c][~hit] = 0.0

        # ---- drag, Coriolis, totals, integration
        mass, inert = self._props(r1, h1)
        fx, fy, m = acc["fcx"] + acc["fbx"] + W["fx"], acc["fcy"] + acc["fby"] + W["fy"], \
            acc["mc"] + acc["mb"] + W["m"]
        body = [np.zeros(n), np.zeros(n)]
        for rho, Cd, Cs, hf, sc, (wu, wv), slow in ((p.rhoair, p.Cdair, p.Csair, ha * h1, sca, wind[:2], 1e-2),
                                                    (p.rhowater, p.Cdwater, p.Cswater, hw * h1, scw, wind[2:], 1e-3)):
            du, dv = wu - u, wv - v
            an = np.sqrt(du * du + dv * dv)
            lg = np.log(hf / p.z0w) / math.log(10.0 / p.z0w)
            form = rho * Cd * hf * r1 * an * lg * lg * sc * p.pi / 2
            skin = np.where(an == 0, 0.0, rho * p.pi * r1 * r1 * Cs / an * (an * an + r1 * r1 * om * om / 4))
            body[0] = body[0] + (form + skin) * du
            body[1] = body[1] + (form + skin) * dv
            m = m - np.where(an < slow, 2 * p.pi / 5 * r1 ** 5 * rho * Cs * om * np.abs(om),
                             0.75 * p.pi * rho * Cs * an * om * r1 ** 4)
        cor = 2 * mass * 7.2921e-5 * p.sin_lat
        fx, fy = fx + body[0] + cor * v, fy + body[1] - cor * u
        u1, v1, om1 = u + fx / mass * dt, v + fy / mass * dt, om + m / inert * dt
        x1, y1 = x + u1 * dt, y + v1 * dt
        if self.px:
            x1 = np.where(x1 < 0, x1 + p.nx, np.where(x1 >= p.nx, x1 - p.nx, x1))
        if self.py:
            y1 = np.where(y1 < 0, y1 + p.ny, np.where(y1 >= p.ny, y1 - p.ny, y1))
        if diag:
            per = lambda a, t: np.where(t != 0, a / t, 0.0)  # noqa: E731
            self.diag = {"tfx": fx, "tfy": fy, "fcx": acc["fcx"], "fcy": acc["fcy"], "fbx": acc["fbx"],
                         "fby": acc["fby"], "m": m, "mc": acc["mc"], "mb": acc["mb"],
                         "tsigxx": acc["sxx"] + W["sxx"] + body[0] * r1, "tsigyy": acc["syy"] + W["syy"] + body[1] * r1,
                         "tsigxy": acc["sxy"] + W["sxy"], "tsigyx": acc["syx"] + W["syx"],
                         "tp": per(acc["pc"], acc["tac"]) + per(acc["pb"], acc["tab"]) + per(W["p"], W["ta"])}
        self.s = {"x": x1, "y": y1, "u": u1, "v": v1, "r": r1, "h": h1, "theta": S["theta"] + om1 * dt, "omega": om1}

    def _walls(self, k, horizontal, far, pos, edge, r1, h1, W):
        p, S = self.p, self.s
        u, v, om, r, h = S["u"][k], S["v"][k], S["omega"][k], r1[k].copy(), h1[k].copy()
        sg = 1.0 if far else -1.0
        c, s = (sg, 0.0) if horizontal else (0.0, sg)
        hist = ("t2", "th2") if horizontal else ("t1", "th1")
        mass, _ = self._props(r, h)
        veln, velt = -u * c - v * s, u * s - v * c - om * r
        dn = (r + pos[k] - edge) if far else (r - pos[k])
        dr = 2 * np.sqrt(r * r - (r - dn) ** 2)
        dtb, thb = self.wall[hist[0]][k] - velt * p.dt, self.wall[hist[1]][k] - om * p.dt
        knc = p.pi * p.ec * h * self._fit(dn * r / (2 * h * h))

        def damp(kn, m):
            ktc = 6 * p.gc / p.ec * kn
            gn = -p.beta * np.sqrt(4 * kn * m)
            return ktc, kn * dr * dr / 12, gn, -2 * p.beta * np.sqrt(2.0 / 3.0 * ktc * m), gn * dr * dr / 12
        ktc, krc, gn, gt, gr = damp(knc, mass)
        fn = np.maximum(knc * dn - gn * veln, 0.0)
        rs, hs = r, h
        if p.ridging:
            pl = p.sigmanc_crit * h <= fn / dr / h
            cap = p.sigmanc_crit * h * h * dr
            ktc, krc, gn, gt, gr = (np.where(pl, b, a) for a, b in
                                    zip((ktc, krc, gn, gt, gr), damp(cap / dn, 0.0)))
            fn = np.where(pl, np.minimum(fn, cap), fn)
            vol = np.maximum((r * r * np.arcsin(dr / 2 / r) - dr * (r - dn) / 2) * h, 0.0)
            a, b = self._grow(r, h, vol)
            rs, hs = np.where(pl, a, r), np.where(pl, b, h)
            dr = np.where(pl, 2 * np.sqrt(rs * rs - (rs - dn) ** 2), dr)
        ft = ktc * dtb - gt * velt
        slip = np.abs(ft) > p.friction_coeff * np.abs(fn)
        ft = np.where(slip, -(p.friction_coeff * np.abs(fn) * np.copysign(1.0, velt)), ft)
        if p.slipping:
            dtb = np.where(slip, (ft + gt * velt) / ktc, dtb)
        roll = np.where(np.abs(thb) > 2 * np.abs(fn) / knc / dr, 0.0, krc * thb - gr * om)
        W["fx"][k] += -fn * c + ft * s
        W["fy"][k] += -fn * s - ft * c
        W["m"][k] += -roll - rs * ft
        q = np.sqrt(fn * fn + ft * ft) * rs
        W["sxx"][k], W["syy"][k], W["sxy"][k], W["syx"][k] = -q * c * c, -q * s * s, -q * c * s, -q * s * c
        W["ta"][k] += dr * hs
        W["p"][k] -= fn * dr * hs
        r1[k], h1[k] = rs, hs
        self.wall[hist[0]][k], self.wall[hist[1]][k] = dtb, thb
