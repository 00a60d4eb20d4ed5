"""The x-sort, the adaptDt median, the division count and the colony radius of
a step against numpy, at the sizes where their kernels change form (a tile of
keys, a block's 32 rows, the one-block scan, the largest colony sorted by
counting) and with many equal keys.  The cells stand apart, so nothing moves
and a step only grows, divides and sorts them; results are exact."""
from __future__ import annotations

import numpy as np
import pytest

from pcc_b200 import abi
from pcc_b200.device import Colony

pytestmark = pytest.mark.gpu


def apart(n: int, columns: int, seed: int) -> dict:
    """n cells on a lattice 4 apart, `columns` distinct x, in shuffled order."""
    rng = np.random.default_rng(seed)
    k = rng.permutation(n)
    x, y = 4.0 * (k % columns) - 2.0 * columns, 4.0 * (k // columns) + 0.5
    th = rng.uniform(0, np.pi, n)
    return {"x": x, "y": y, "z": np.zeros(n), "q0": np.cos(th / 2), "q1": np.zeros(n), "q2": np.zeros(n),
            "q3": np.sin(th / 2), "length": rng.uniform(1.0, 1.9, n), "l0": np.ones(n), "diameter": np.full(n, 0.5),
            "age": np.ones(n, np.int32)}


SIZES = [1, 2, 31, 32, 33, 255, 257, 2047, 2048, 2049, 8193, 16383, 16384, 16385, 33000]


def step_of(cells: dict, **over):
    p = abi.default_params(mode=abi.MODE_SOFT, kcc=1000.0, dt=1e-3, ghost_mode=abi.GHOSTS_NONE, **over)
    g = Colony(p)
    g.set_cells(cells)
    st = g.step()
    return p, st, g.get_cells()


def check(cells: dict, st: dict, got: dict, p):
    o = np.argsort(cells["x"], kind="stable")
    np.testing.assert_array_equal(got["x"], cells["x"][o])
    np.testing.assert_array_equal(got["y"], cells["y"][o])
    length = cells["length"][o]
    np.testing.assert_array_equal(got["length"], np.minimum(length + p.dt * length, 2.0))
    speed = np.sort(length)
    n = len(speed)
    med = speed[n // 2] if n % 2 else 0.5 * (speed[n // 2 - 1] + speed[n // 2])
    want = min(max(p.dt * 0.99 + 0.01 * (0.5e-3 / med), 0.9 * p.dt), 1.1 * p.dt)
    assert abs(st["dt_next"] - want) <= 1e-15 * want
    half = got["length"] / 2 - 0.25
    tx, ty = 1 - 2 * got["q3"] ** 2, 2 * got["q0"] * got["q3"]
    r = np.hypot(got["x"] + tx * half, got["y"] + ty * half).max()
    assert abs(st["colony_radius"] - r) <= 1e-13 * r


@pytest.mark.parametrize("n", SIZES)
def test_order_median_and_radius(n):
    cells = apart(n, max(1, int(np.sqrt(n))), n)
    p, st, got = step_of(cells)
    check(cells, st, got, p)


@pytest.mark.parametrize("n", [3000, 17001])
def test_one_column(n):
    """Every key equal: the order is the order of upload."""
    cells = apart(n, 1, n)
    p, st, got = step_of(cells)
    check(cells, st, got, p)


@pytest.mark.parametrize("n,dividing", [(1, 1), (300, 7), (8200, 8200), (33000, 1000)])
def test_division_count(n, dividing):
    """Cells that reach twice their birth length divide in the next step."""
    cells = apart(n, max(1, int(np.sqrt(n))), n)
    cells["length"][:] = 1.2
    cells["length"][np.random.default_rng(5).permutation(n)[:dividing]] = 1.9995
    p = abi.default_params(mode=abi.MODE_SOFT, kcc=1000.0, dt=1e-3, fixed_dt=1, ghost_mode=abi.GHOSTS_NONE)
    g = Colony(p)
    g.set_cells(cells)
    first, second = g.step(), g.step()
    assert first["n_divided"] == 0 and first["n_cells"] == n
    assert second["n_divided"] == dividing and second["n_cells"] == n + dividing
