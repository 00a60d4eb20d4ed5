"""Colonies whose cells have very different numbers of contacts: a knot of
overlapping cells beside a field of sparse ones, so that an even share of the
contacts' weight leaves one block of the on-chip BBPGD solver with about twice
the mean.  Each entry: cells of the knot, sparse cells, knot cells per unit
area, and for the FP64, mixed and 3D forms the solver's form and the groups of
16 cells that find no room in their block's shared memory."""
from __future__ import annotations

import numpy as np

UNEVEN = [
    ((160, 900, 100.0), [("cluster", 1), ("cluster", 0), ("cluster", 3)]),
    ((250, 1500, 12.0), [("cluster", 7), ("cluster", 0), ("grid", 0)]),
    ((300, 2000, 30.0), [("grid", 0), ("cluster", 6), ("grid", 0)]),
    ((300, 3000, 40.0), [("grid", 0), ("grid", 0), ("grid", 6)]),
    ((800, 28000, 30.0), [("grid", 58), ("grid", 25), ("streaming", 0)]),
]


def uneven(knot: int, sparse: int, density: float, seed: int = 3) -> dict:
    rng = np.random.default_rng(seed)
    w, side = 12.0, np.sqrt(sparse / 0.45)
    h = knot / density / w
    x = np.concatenate([rng.uniform(0, w, knot), 14 + rng.uniform(0, side, sparse)])
    y = np.concatenate([rng.uniform(-h / 2, h / 2, knot), rng.uniform(-side / 2, side / 2, sparse)])
    n = knot + sparse
    th = rng.uniform(0, np.pi, n)
    o = np.argsort(x, kind="stable")
    return {"x": x[o], "y": y[o], "z": np.zeros(n), "q0": np.cos(th / 2), "q1": np.zeros(n), "q2": np.zeros(n),
            "q3": np.sin(th / 2), "length": rng.uniform(1.0, 1.9, n), "l0": np.ones(n),
            "diameter": np.full(n, 0.5), "age": np.ones(n, np.int32)}
