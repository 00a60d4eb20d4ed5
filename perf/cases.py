"""Cases by which the speed of the collision hot path is measured.

A user of this library grows colonies of rod-shaped cells: one colony stepped
for a long time (hard or soft model, FP64 or mixed precision), one solver call
per step behind the reference's driver (state in, state out), several colonies
in lockstep, or a queue of colony jobs.  The cases below are those uses, from
a seedling of some twenty cells, whose step is launches and latency, to the
grown colony of radius 260 (302,180 cells), whose step is memory traffic.

The states are pieces of the colony that this library grew from one cell to
R = 260 (the benchmark's start state): the cells nearest to a centre drawn
from the seed, as many as a colony of `radius` has, turned by an angle drawn
from the seed, in x order.  They carry the packing, the orientations, the
lengths and the residual overlaps of a grown colony.  Its angles are stored in
32 bits, so sisters can be exactly parallel there, which leaves their contact
point to rounding: each cell is turned by up to JITTER more.  Soft colonies
are denser than hard ones (their cells overlap under pressure), so their
pieces are squeezed by SQUEEZE.
"""
from __future__ import annotations

import ctypes as C
import math
from functools import lru_cache

import numpy as np
import torch

import pcc_pkg

pcc_pkg.load_package()

from pcc_b200 import abi, device  # noqa: E402

GROWN = pcc_pkg.PKG_DIR / "data" / "colony_r260_seed0.npz"
FULL = 260.0  # radius of that colony
CELLS_PER_R2 = 4.47  # its cells per radius^2
SQUEEZE = 0.85
JITTER = 1e-3
KCC_SOFT = 1333.3333333333333  # 4/3 E at E = 1e3
DT_HARD, DT_SOFT = 1e-3, 3e-5
STATE = ("x", "y", "z", "q0", "q1", "q2", "q3", "length", "l0", "diameter", "ldot", "impedance", "stress")
CELL_BYTES = 8 * (len(STATE) + 12) + 4  # the state of one cell, force and velocity among it


def listed() -> list[dict]:
    return [
        # a job's first hours: some twenty cells, every step a string of small launches
        dict(name="hard_seedling", kind="run", model="hard", mixed=False, radius=2.5, steps=20, adapt=False),
        # a small colony of a parameter sweep, CFL-adaptive time step
        dict(name="hard_r10", kind="run", model="hard", mixed=False, radius=10.0, steps=5, adapt=True),
        # the plain method's single colony at its end, R = 20, fixed time step
        dict(name="hard_r20", kind="run", model="hard", mixed=False, radius=20.0, steps=3, adapt=False),
        # a larger colony of a sweep in mixed precision (an odd radius, a ragged count)
        dict(name="hard_mixed_r45", kind="run", model="hard", mixed=True, radius=45.3, steps=2, adapt=True),
        # the solver behind the reference's driver: state in, one solver call, state and constraint set out
        dict(name="hard_call_r100", kind="call", model="hard", mixed=False, radius=100.0, steps=1, adapt=False),
        # the largest: a whole step of the grown colony in mixed precision, state in and out as end to end
        dict(name="hard_mixed_r260", kind="run", model="hard", mixed=True, radius=260.0, steps=1, adapt=True),
        # Brownian kicks out of the plane (monolayer off): the three-dimensional solver
        dict(name="hard_3d_r15", kind="run", model="hard3d", mixed=False, radius=15.0, steps=4, adapt=False),
        # the soft model's single colony at its end; its steps are short and hundreds of thousands
        dict(name="soft_r20", kind="run", model="soft", mixed=False, radius=20.0, steps=20, adapt=False),
        # a large soft colony, where a step is memory traffic
        dict(name="soft_r120", kind="run", model="soft", mixed=False, radius=120.0, steps=4, adapt=False),
        # the soft assembly on a host's own device buffers
        dict(name="soft_forces_37k", kind="forces", radius=77.7),
        # an uneven sweep in lockstep
        dict(name="batch_8", kind="batch", colonies=8, r_min=4.0, r_max=25.0, steps=2),
        # a queue of jobs from single cells, four hard to one soft, eight in flight
        dict(name="serve_10", kind="serve", jobs=10, slots=8, steps=60),
    ]


def draw(rng) -> dict:
    def log(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 2)

    kind = rng.choice(["hard", "hard", "hard", "call", "hard3d", "soft", "soft", "forces", "batch", "serve"])
    if kind == "hard":
        r = log(2.0, 180.0)
        return dict(kind="run", model="hard", mixed=rng.random() < 0.5, radius=r,
                    steps=max(1, min(20, int(60 / r))), adapt=rng.random() < 0.5)
    if kind == "call":
        return dict(kind="call", model="hard", mixed=rng.random() < 0.5, radius=log(5.0, 130.0), steps=1, adapt=False)
    if kind == "hard3d":
        return dict(kind="run", model="hard3d", mixed=False, radius=log(3.0, 40.0), steps=rng.randint(2, 4),
                    adapt=False)
    if kind == "soft":
        r = log(2.0, 150.0)
        return dict(kind="run", model="soft", mixed=False, radius=r, steps=max(2, min(20, int(400 / r))), adapt=False)
    if kind == "forces":
        return dict(kind="forces", radius=log(2.0, 100.0))
    if kind == "batch":
        return dict(kind="batch", colonies=rng.randint(2, 10), r_min=round(rng.uniform(2.0, 5.0), 2),
                    r_max=round(rng.uniform(10.0, 30.0), 2), steps=rng.randint(1, 3))
    return dict(kind="serve", jobs=rng.randint(4, 14), slots=rng.randint(2, 8), steps=rng.randint(20, 80))


# ---------------------------------------------------------------- inputs
@lru_cache(maxsize=1)
def _grown() -> dict:
    with np.load(GROWN) as d:
        return {k: d[k].astype(np.float64) for k in ("x", "y", "theta", "length", "l0", "diameter")} | {
            "age": d["age"].astype(np.int32)}


def _count(radius: float, squeeze: float = 1.0) -> int:
    return min(_grown()["x"].size, int(CELLS_PER_R2 * (radius / squeeze) ** 2))


def _room(n: int) -> int:
    """Cells that the result buffers of a colony of n cells hold (it divides)."""
    return n + n // 4 + 64


def _piece(radius: float, rng: np.random.Generator, squeeze: float = 1.0) -> dict:
    """The cells nearest to a drawn centre, turned by a drawn angle, squeezed
    towards the centre, in x order."""
    g = _grown()
    take = radius / squeeze
    off = max(0.0, FULL - take) * math.sqrt(rng.random())
    at = rng.uniform(0.0, 2.0 * math.pi)
    turn = rng.uniform(0.0, 2.0 * math.pi)
    dx, dy = g["x"] - off * math.cos(at), g["y"] - off * math.sin(at)
    n = _count(radius, squeeze)
    k = np.argpartition(dx * dx + dy * dy, n - 1)[:n]
    c, s = math.cos(turn), math.sin(turn)
    x, y = squeeze * (c * dx[k] - s * dy[k]), squeeze * (s * dx[k] + c * dy[k])
    o = np.argsort(x, kind="stable")
    k = k[o]
    th = g["theta"][k] + turn + rng.uniform(-JITTER, JITTER, n)
    return {"x": x[o], "y": y[o], "z": np.zeros(n), "q0": np.cos(th / 2), "q1": np.zeros(n), "q2": np.zeros(n),
            "q3": np.sin(th / 2), "length": g["length"][k], "l0": g["l0"][k], "diameter": g["diameter"][k],
            "age": g["age"][k]}


def _params(case: dict, seed: int):
    model = case["model"]
    kw = dict(seed=seed, fixed_dt=0 if case["adapt"] else 1, dt=DT_HARD, mode=abi.MODE_HARD,
              precision=abi.PRECISION_MIXED if case["mixed"] else abi.PRECISION_FP64)
    if case["adapt"]:
        kw["dt_cap"] = DT_HARD
    if model == "hard3d":
        kw.update(temperature=0.5, monolayer=0)
    if model == "soft":
        kw.update(mode=abi.MODE_SOFT, dt=DT_SOFT, kcc=KCC_SOFT)
    return abi.default_params(**kw)


class Buffers:
    """Pinned host arrays of `cap` cells in the layout that the ABI takes."""

    def __init__(self, cap: int):
        pin = torch.cuda.is_available()
        self.cap = cap
        self.t = {f: torch.zeros(cap, dtype=torch.float64, pin_memory=pin) for f in STATE}
        self.t["force"] = torch.zeros((cap, 6), dtype=torch.float64, pin_memory=pin)
        self.t["velocity"] = torch.zeros((cap, 6), dtype=torch.float64, pin_memory=pin)
        self.t["age"] = torch.zeros(cap, dtype=torch.int32, pin_memory=pin)
        self.t["num_constraints"] = torch.zeros(cap, dtype=torch.int32, pin_memory=pin)
        self.struct = abi.Cells()
        for f, v in self.t.items():
            kind = C.c_int if v.dtype == torch.int32 else C.c_double
            setattr(self.struct, f, C.cast(v.data_ptr(), C.POINTER(kind)))

    def fill(self, cells: dict) -> "Buffers":
        for f, v in cells.items():
            self.t[f][: len(v)] = torch.from_numpy(np.ascontiguousarray(v))
        return self



def _colony_state(col, cells: dict, dt: float) -> dict:
    n = len(cells["x"])
    return {"col": col, "n": n, "dt": dt, "in": Buffers(n).fill(cells), "out": Buffers(_room(n))}


def _jobs(case: dict, seed: int) -> list[dict]:
    rng = np.random.default_rng(seed)
    jobs = []
    for k in range(case["jobs"]):
        rate = float(rng.uniform(0.5, 1.5))  # growth rate
        if k % 5 == 4:
            p = abi.default_params(mode=abi.MODE_SOFT, dt=DT_SOFT, fixed_dt=1, kcc=KCC_SOFT)
        else:
            p = abi.default_params(mode=abi.MODE_HARD, dt=DT_HARD, dt_cap=DT_HARD, precision=abi.PRECISION_MIXED)
        p.seed, p.tau = int(rng.integers(1 << 31)), 1.0 / rate
        if k % 5 != 4:
            p.dt, p.dt_cap = 2e-2, 2e-2  # the early steps, a division every few tens of steps
        jobs.append({"params": p, "end_radius": float(np.exp(rng.uniform(np.log(10.0), np.log(150.0)))),
                     "arrival_s": 0.0, "max_steps": case["steps"]})
    return jobs


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("run", "call"):
        cells = _piece(case["radius"], rng, SQUEEZE if case["model"] == "soft" else 1.0)
        p = _params(case, seed)
        p.capacity_hint = int(1.2 * len(cells["x"])) + 64
        state = {"case": case, **_colony_state(device.Colony(p), cells, p.dt)}
        if kind == "call":
            state["constraints"] = abi.ContactArrays(24 * len(cells["x"]))
        return state
    if kind == "batch":
        one = dict(model="hard", mixed=True, adapt=True)
        radii = np.geomspace(case["r_min"], case["r_max"], case["colonies"])
        b = device.Batch([_params(one, seed + k) for k in range(case["colonies"])])
        return {"case": case, "batch": b, "states": [_colony_state(b[k], _piece(float(r), rng), DT_HARD)
                                                     for k, r in enumerate(radii)]}
    if kind == "serve":
        return {"case": case, "jobs": _jobs(case, seed)}
    # forces: contacts and diameters in the caller's own device buffers
    f = device.load_library().pcc_soft_forces_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p] * 8 + [C.c_size_t, C.c_void_p, C.c_size_t, C.c_double] + [C.c_void_p] * 3
    cells, con = _forces_input(case, seed)
    n = len(cells["x"])
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in con.items()}
    return {"case": case, "call": f, "n": n, "m": int(con["sd"].size), "dev": dev,
            "diameter": torch.from_numpy(cells["diameter"]).cuda(),
            "force": torch.zeros((n, 6), dtype=torch.float64, device="cuda"),
            "stress": torch.zeros(n, dtype=torch.float64, device="cuda")}


# ---------------------------------------------------------------- one pass
_STATS = ("relcp_iterations", "bbpgd_iterations", "residual", "max_overlap", "n_constraints", "n_cells", "n_divided",
          "dt_next", "colony_radius")


def _stats(st: dict, keys=_STATS) -> dict:
    return {k: st[k] for k in keys}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        # from a checkpoint (state and time step), some steps on the device, the state read back
        col = state["col"]
        col.upload(state["in"], state["n"])
        col.dt = state["dt"]
        _, cell_steps, last = col.run(math.inf, case["steps"])
        n = col.download(state["out"])
        return {"n": n, "cells": state["out"].t, "cell_steps": cell_steps, "last": _stats(last)}
    if kind == "call":
        col = state["col"]
        col.upload(state["in"], state["n"])
        st = col.solve(state["dt"], 1)
        n = col.download(state["out"])
        con, m = state["constraints"], C.c_size_t(0)
        rc = col.lib.pcc_get_constraints(col.h, C.byref(con.struct), con.cap, C.byref(m))
        if rc != abi.PCC_OK:
            raise device.PccError(rc, f"pcc_get_constraints: {abi.STATUS_NAMES.get(rc, rc)}")
        return {"n": n, "m": m.value, "cells": state["out"].t, "constraints": con.arrays,
                "last": _stats(st, ("relcp_iterations", "bbpgd_iterations", "residual", "max_overlap",
                                    "n_constraints"))}
    if kind == "batch":
        for s in state["states"]:
            s["col"].upload(s["in"], s["n"])
            s["col"].dt = s["dt"]
        for _ in range(case["steps"]):
            last = state["batch"].step()
        out = []
        for s in state["states"]:
            n = s["col"].download(s["out"])
            out.append({"n": n, **{k: s["out"].t[k] for k in ("x", "y", "q0", "q3", "length")}})
        return {"cells": out, "bbpgd": np.array([st["bbpgd_iterations"] for st in last])}
    if kind == "serve":
        res, _ = device.serve(state["jobs"], slots=case["slots"])
        return {k: np.array([r[k] for r in res])
                for k in ("steps", "cells", "cell_steps", "bbpgd_iterations", "checksum", "radius", "dt")}
    d = state["dev"]
    rc = state["call"](d["gid_i"].data_ptr(), d["gid_j"].data_ptr(), d["sd"].data_ptr(), d["normal"].data_ptr(),
                       d["r_i"].data_ptr(), d["r_j"].data_ptr(), d["stress_i"].data_ptr(), d["stress_j"].data_ptr(),
                       state["m"], state["diameter"].data_ptr(), state["n"], KCC_SOFT, state["force"].data_ptr(),
                       state["stress"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if rc != abi.PCC_OK:
        raise device.PccError(rc, f"pcc_soft_forces_noalloc: {abi.STATUS_NAMES.get(rc, rc)}")
    return {"force": state["force"], "stress": state["stress"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case: dict) -> dict:
    """Bytes: the state read and written once per step (the constraints of a
    step come from it and need not leave the chip).  Operations: per cell and
    step some 30 candidate pairs of 20 operations, 5 contacts of 150 and, in
    the hard model, at least 10 iterations over 5 constraints of 40 (the
    residual is tested every tenth)."""
    kind = case["kind"]
    if kind == "forces":
        n = CELLS_PER_R2 * (case["radius"] / SQUEEZE) ** 2
        return {"bytes": n * (8 + 56) + 4.5 * n * (8 + 4 * 24), "flops": 4.5 * n * 60}
    if kind == "batch":
        radii = np.geomspace(case["r_min"], case["r_max"], case["colonies"])
        cell_steps, hard = case["steps"] * CELLS_PER_R2 * float((radii * radii).sum()), True
    elif kind == "serve":
        cell_steps, hard = 2.0 * case["jobs"] * case["steps"], True
    else:
        r = case["radius"] / (SQUEEZE if case["model"] == "soft" else 1.0)
        cell_steps, hard = case["steps"] * CELLS_PER_R2 * r * r, case["model"] != "soft"
    return {"bytes": 2.0 * CELL_BYTES * cell_steps, "flops": cell_steps * (600 + 750 + (2000 if hard else 0))}


# ---------------------------------------------------------------- the same in plain 64-bit numpy
def _pairs(x, y, reach: float):
    """Index pairs i < j whose centres are closer than `reach`."""
    bx, by = np.floor(x / reach).astype(np.int64), np.floor(y / reach).astype(np.int64)
    bx, by = bx - bx.min() + 1, by - by.min() + 1
    w = int(by.max()) + 2
    key = bx * w + by
    o = np.argsort(key, kind="stable")
    sk = key[o]
    out = []
    for d in (-w - 1, -w, -w + 1, -1, 0, 1, w - 1, w, w + 1):
        lo, hi = np.searchsorted(sk, key + d, "left"), np.searchsorted(sk, key + d, "right")
        cnt = hi - lo
        i = np.repeat(np.arange(x.size), cnt)
        j = o[np.repeat(lo - np.concatenate(([0], np.cumsum(cnt)[:-1])), cnt) + np.arange(i.size)]
        k = (i < j) & ((x[i] - x[j]) ** 2 + (y[i] - y[j]) ** 2 < reach * reach)
        out.append(np.stack([i[k], j[k]]))
    i, j = np.concatenate(out, axis=1)
    o = np.lexsort((j, i))
    return i[o], j[o]


def _contacts(c: dict, tol: float) -> dict:
    """Contacts i < j of a planar colony with separation <= tol: closest points
    of the two axis segments, the nearest of the interior solution and the four
    end-to-segment solutions."""
    x, y = c["x"], c["y"]
    tx, ty = c["q0"] ** 2 - c["q3"] ** 2, 2.0 * c["q0"] * c["q3"]
    half = c["length"] / 2 - c["diameter"] / 2
    i, j = _pairs(x, y, 2.0 + max(tol, 0.0))
    ux, uy, vx, vy = 2 * half[i] * tx[i], 2 * half[i] * ty[i], 2 * half[j] * tx[j], 2 * half[j] * ty[j]
    px, py = x[i] - half[i] * tx[i], y[i] - half[i] * ty[i]
    qx, qy = x[j] - half[j] * tx[j], y[j] - half[j] * ty[j]
    wx, wy = px - qx, py - qy
    a, b, cc = ux * ux + uy * uy, ux * vx + uy * vy, vx * vx + vy * vy
    d, e = ux * wx + uy * wy, vx * wx + vy * wy
    det = a * cc - b * b
    safe = np.where(det > 0, det, 1.0)
    s0, t0 = (b * e - cc * d) / safe, (a * e - b * d) / safe
    inside = (det > 0) & (s0 >= 0) & (s0 <= 1) & (t0 >= 0) & (t0 <= 1)
    one, zero = np.ones_like(a), np.zeros_like(a)
    best = np.full(a.shape, np.inf)
    s, t = zero.copy(), zero.copy()
    for cs, ct, ok in ((zero, np.clip(e / cc, 0, 1), one > 0), (one, np.clip((e + b) / cc, 0, 1), one > 0),
                       (np.clip(-d / a, 0, 1), zero, one > 0), (np.clip((b - d) / a, 0, 1), one, one > 0),
                       (s0, t0, inside)):
        d2 = (wx + cs * ux - ct * vx) ** 2 + (wy + cs * uy - ct * vy) ** 2
        k = ok & (d2 < best)
        best[k], s[k], t[k] = d2[k], cs[k], ct[k]
    dist = np.sqrt(best)
    sd = dist - (c["diameter"][i] + c["diameter"][j]) / 2
    k = sd <= tol
    i, j, s, t, sd, dist = i[k], j[k], s[k], t[k], sd[k], dist[k]
    ax, ay = px[k] + s * ux[k], py[k] + s * uy[k]
    bx, by = qx[k] + t * vx[k], qy[k] + t * vy[k]
    nx, ny = (ax - bx) / dist, (ay - by) / dist
    mx, my = (ax + bx) / 2, (ay + by) / 2
    z = np.zeros_like(sd)
    return {"gid_i": i.astype(np.int32), "gid_j": j.astype(np.int32), "sd": sd, "normal": np.stack([nx, ny, z], 1),
            "r_i": np.stack([mx - x[i], my - y[i], z], 1), "r_j": np.stack([mx - x[j], my - y[j], z], 1),
            "stress_i": 0.5 * np.abs(nx * tx[i] + ny * ty[i]), "stress_j": 0.5 * np.abs(nx * tx[j] + ny * ty[j])}


def _forces_input(case: dict, seed: int):
    cells = _piece(case["radius"], np.random.default_rng(seed), SQUEEZE)
    return cells, _contacts(cells, 0.0)


def _hertz(c: dict, con: dict, copies) -> tuple:
    """Force (x, y), torque (z) and stress per cell of the overlapping contacts."""
    n = c["x"].size
    i, j = con["gid_i"], con["gid_j"]
    over = np.maximum(-con["sd"], 0.0)
    r1, r2 = c["diameter"][i] / 2, c["diameter"][j] / 2
    fe = copies * KCC_SOFT * np.sqrt(r1 * r2 / (r1 + r2)) * over ** 1.5
    fx, fy = con["normal"][:, 0] * fe, con["normal"][:, 1] * fe

    def per_cell(vi, vj):
        return np.bincount(i, vi, n) + np.bincount(j, vj, n)

    tz = per_cell(con["r_i"][:, 0] * fy - con["r_i"][:, 1] * fx, -(con["r_j"][:, 0] * fy - con["r_j"][:, 1] * fx))
    return per_cell(fx, -fx), per_cell(fy, -fy), tz, per_cell(con["stress_i"] * fe, con["stress_j"] * fe)


def _self_ghost(x, y):
    """Cells that the single-rank decomposition also sends to itself: at least
    8 from the origin and within 2.5 of the sector edge at angle 0."""
    ang = np.degrees(np.arctan2(y, x))
    ang = np.where(ang < 0, ang + 360.0, ang)
    r = np.hypot(x, y)
    lo = np.where(ang > 180.0, ang - 360.0, ang)
    hi = np.where(360.0 - ang > 180.0, -ang, 360.0 - ang)
    near = np.where((lo >= 0) & (hi >= 0), 0.0, r * np.sin(np.radians(np.minimum(np.abs(lo), np.abs(hi)))))
    return (r >= 8.0) & (near < 2.5)


def _left_length(seed: int, k: int, length: float) -> float:
    """Length of the left daughter of a colony's k-th division: uniform in
    [0.98, 1.02] times half, from an MT19937 seeded by a splitmix64 finaliser."""
    m64 = (1 << 64) - 1
    z = (seed + 0x9E3779B97F4A7C15 * (k + 1)) & m64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m64
    g = np.random.MT19937()
    g._legacy_seeding((z ^ (z >> 31)) & 0xFFFFFFFF)
    lo, hi = (int(v) for v in g.random_raw(2))
    u = (float(lo) + float(hi) * 4294967296.0) / 18446744073709551616.0
    return u * (1.02 * length / 2 - 0.98 * length / 2) + 0.98 * length / 2


def _soft_steps(c: dict, steps: int, seed: int) -> dict:
    xi, lam, tau, dt = 1.0, 1e-2, 1.0, DT_SOFT
    c = {k: np.array(v) for k, v in c.items()}
    drawn = 0
    for _ in range(steps):
        who = np.nonzero(c["length"] >= 2.0 * c["l0"])[0]
        if who.size:
            left = np.array([_left_length(seed, drawn + k, float(c["length"][w])) for k, w in enumerate(who)])
            drawn += who.size
            right = c["length"][who] - left
            tx, ty = c["q0"][who] ** 2 - c["q3"][who] ** 2, 2.0 * c["q0"][who] * c["q3"][who]
            new = {k: v[who].copy() for k, v in c.items()}
            new["x"], new["y"], new["length"] = new["x"] + tx * right / 2, new["y"] + ty * right / 2, right
            c["x"][who] -= tx * left / 2
            c["y"][who] -= ty * left / 2
            c["length"][who] = left
            c["age"][who] += 1
            new["age"] = new["age"] + 1
            c = {k: np.concatenate([v, new[k]]) for k, v in c.items()}
        o = np.argsort(c["x"], kind="stable")
        c = {k: v[o] for k, v in c.items()}
        con = _contacts(c, 0.0)
        fx, fy, tz, sig = _hertz(c, con, 1 + _self_ghost(c["x"], c["y"])[con["gid_j"]])
        ml, mr = 1.0 / (c["length"] * xi), 12.0 / (c["length"] ** 3 * xi)
        ux, uy, wz = ml * fx, ml * fy, mr * tz
        c["x"], c["y"] = c["x"] + dt * ux, c["y"] + dt * uy
        q0, q3 = c["q0"] - dt * 0.5 * c["q3"] * wz, c["q3"] + dt * 0.5 * c["q0"] * wz
        nrm = np.sqrt(q0 * q0 + q3 * q3)
        c["q0"], c["q3"] = q0 / nrm, q3 / nrm
        imp = np.exp(-lam * sig)
        ldot = c["length"] / tau * imp
        c["length"] = np.minimum(c["length"] + dt * ldot, 2.0 * c["l0"])
    z = np.zeros_like(fx)
    return {"x": c["x"], "y": c["y"], "z": z, "q0": c["q0"], "q1": z, "q2": z, "q3": c["q3"], "length": c["length"],
            "l0": c["l0"], "diameter": c["diameter"], "ldot": ldot, "impedance": imp, "stress": sig,
            "force": np.stack([fx, fy, z, z, z, tz], 1), "velocity": np.stack([ux, uy, z, z, z, wz], 1)}


def exact(case: dict, seed: int):
    """The soft model's results.  The hard model has no such value: its solver
    stops anywhere below the tolerance, and over hundreds of iterations of a
    method that is not monotone two orders of summation end at two such points."""
    if case["kind"] == "forces":
        c, con = _forces_input(case, seed)
        fx, fy, tz, sig = _hertz(c, con, 1)
        z = np.zeros_like(fx)
        return {"force": np.stack([fx, fy, z, z, z, tz], 1), "stress": sig}
    if case["kind"] == "run" and case["model"] == "soft":
        c = _piece(case["radius"], np.random.default_rng(seed), SQUEEZE)
        room = _room(len(c["x"]))
        cells = {k: np.concatenate([v, np.zeros((room - len(v), *v.shape[1:]))])
                 for k, v in _soft_steps(c, case["steps"], seed).items()}
        return {"n": None, "cells": {**cells, "age": None, "num_constraints": None}, "cell_steps": None, "last": None}
    return None
