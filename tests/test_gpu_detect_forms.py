"""Contact lists against the C oracle, bit for bit, where the detection changes
form: group and block edges of the pair passes, candidate lists that overflow
(the stencil emit), colonies whose bins are not the assumed box around the
radius (out of the plane, a chain too long for it, a cell whose centre lies
beyond it), and a solve of each."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import normalized_contacts
from oracles import OracleColony
from pcc_b200 import abi
from pcc_b200.device import Colony

pytestmark = pytest.mark.gpu


def cells_at(x, y, z, rng, lo=1.0, hi=2.0, tilt=0.0) -> dict:
    n = len(x)
    th, ph = rng.uniform(0, 2 * np.pi, n), tilt * rng.uniform(-1, 1, n)
    # rotation about z, then a small one about y
    q = np.stack([np.cos(th / 2) * np.cos(ph / 2), -np.sin(th / 2) * np.sin(ph / 2),
                  np.cos(th / 2) * np.sin(ph / 2), np.sin(th / 2) * np.cos(ph / 2)])
    o = np.argsort(x, kind="stable")
    return {"x": np.asarray(x)[o], "y": np.asarray(y)[o], "z": np.asarray(z)[o], "q0": q[0], "q1": q[1], "q2": q[2],
            "q3": q[3], "length": rng.uniform(lo, hi, n), "l0": np.ones(n), "diameter": np.full(n, 0.5),
            "age": np.ones(n, np.int32)}


def scattered(n, seed, spread=0.8, **kw):
    rng = np.random.default_rng(seed)
    r = spread * np.sqrt(n)
    return cells_at(rng.uniform(-r, r, n), rng.uniform(-r, r, n), np.zeros(n), rng, **kw)


def crowd(n, seed):
    rng = np.random.default_rng(seed)
    return cells_at(rng.uniform(-0.6, 0.6, n), rng.uniform(-0.6, 0.6, n), np.zeros(n), rng)


def solid(n, seed):
    rng = np.random.default_rng(seed)
    r = 1.1 * n ** (1 / 3)
    return cells_at(*rng.uniform(-r, r, (3, n)), rng, tilt=1.0)


def chain(n, seed):
    rng = np.random.default_rng(seed)
    return cells_at(1.3 * np.arange(n), rng.uniform(-0.1, 0.1, n), np.zeros(n), rng)


def overhang(n, seed):
    """One long cell whose leading end points inwards: its centre is outside
    the colony radius by more than any grown cell's can be."""
    c = scattered(n, seed)
    c["x"][-1], c["y"][-1], c["length"][-1] = 60.0, 0.0, 30.0
    c["q0"][-1], c["q3"][-1] = 0.0, 1.0
    return c


COLONIES = [(f"scattered{n}", scattered(n, n)) for n in (1, 2, 3, 31, 32, 33, 255, 257, 2100)] + [
    ("crowd40", crowd(40, 1)), ("crowd90", crowd(90, 2)), ("solid300", solid(300, 3)), ("chain900", chain(900, 4)),
    ("overhang50", overhang(50, 5)), ("ghosts", scattered(1500, 7, spread=0.6))]


@pytest.mark.parametrize("tol", [0.25, 1e-3, 0.0, 0.6])
@pytest.mark.parametrize("name,cells", COLONIES, ids=[n for n, _ in COLONIES])
def test_contacts_match_oracle(name, cells, tol):
    p = abi.default_params()
    g, o = Colony(p), OracleColony(p)
    g.set_cells(cells)
    o.set_cells(cells)
    got, want = normalized_contacts(g.detect(tol, 0)), normalized_contacts(o.detect(tol, 0))
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    if name == "crowd90" and tol > 0:
        assert np.bincount(want["gid_i"]).max() > 32  # the lists overflow


@pytest.mark.parametrize("name", ["scattered257", "solid300", "chain900", "overhang50", "ghosts"])
def test_soft_step_matches_oracle(name):
    """A whole soft step: contacts, per-cell counts and forces."""
    cells = dict(COLONIES)[name]
    p = abi.default_params(mode=abi.MODE_SOFT, kcc=1000.0, dt=1e-6, fixed_dt=1)
    g, o = Colony(p), OracleColony(p)
    for c in (g, o):
        c.set_cells(cells)
    for _ in range(2):
        sg, so = g.step(), o.step()
        assert sg["n_constraints"] == so["n_constraints"] and sg["n_cells"] == so["n_cells"]
    a, b = g.get_cells(), o.get_cells()
    np.testing.assert_array_equal(a["num_constraints"], b["num_constraints"])
    np.testing.assert_allclose(a["force"], b["force"], rtol=1e-9, atol=1e-9)
