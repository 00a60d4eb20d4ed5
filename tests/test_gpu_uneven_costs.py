"""Steps of colonies that a pass was not laid out for cost no more than a few
times an ordinary step of as many cells.  Each bound lies far above what the
step takes (at most 2 times) and far below what a pass quadratic in the cells
takes (20 times and more)."""
from __future__ import annotations

import time

import numpy as np
import pytest

from pcc_b200 import abi
from pcc_b200.device import Colony

pytestmark = pytest.mark.gpu

N = 400_000


def rods(x, y, z, rng) -> dict:
    n = len(x)
    th = rng.uniform(0, np.pi, n)
    return {"x": x, "y": y, "z": z, "q0": np.cos(th / 2), "q1": np.zeros(n), "q2": np.zeros(n), "q3": np.sin(th / 2),
            "length": rng.uniform(1.0, 1.9, n), "l0": np.ones(n), "diameter": np.full(n, 0.5),
            "age": np.ones(n, np.int32)}


def first_and_later(cells: dict) -> tuple[float, float]:
    """Seconds of the first step after an upload and of a later one, the
    quickest of three uploads (the first allocates)."""
    g = Colony(abi.default_params(mode=abi.MODE_SOFT, kcc=1000.0, dt=1e-7, fixed_dt=1, ghost_mode=abi.GHOSTS_NONE))
    first, later = [], []
    for _ in range(3):
        g.set_cells(cells)
        for times in (first, later):
            t = time.perf_counter()
            g.step()
            times.append(time.perf_counter() - t)
    return min(first), min(later)


def test_first_detection_of_a_solid_colony():
    """Its cells lie outside the box of a flat one."""
    rng = np.random.default_rng(1)
    r = N ** (1 / 3)
    first, later = first_and_later(rods(*rng.uniform(-r, r, (3, N)), rng))
    assert first < 8 * later, (first, later)


@pytest.mark.parametrize("columns", [1, 32])
def test_sort_of_a_tall_colony(columns):
    """Its cells share few x."""
    rng = np.random.default_rng(1)
    k = np.arange(N)
    square = int(np.sqrt(N))
    usual = first_and_later(rods(4.0 * (k % square), 4.0 * (k // square), np.zeros(N), rng))
    tall = first_and_later(rods(4.0 * (k % columns), 4.0 * (k // columns), np.zeros(N), rng))
    assert tall[0] < 4 * usual[0] and tall[1] < 4 * usual[1], (tall, usual)


def test_order_of_a_colony_that_crowds_and_spreads():
    """The x-sort on both sides of its change of form, after one another on one context: the order is a stable sort."""
    rng = np.random.default_rng(2)
    n = 40_000
    k = rng.permutation(n)
    g = Colony(abi.default_params(mode=abi.MODE_SOFT, kcc=1000.0, dt=1e-7, fixed_dt=1, ghost_mode=abi.GHOSTS_NONE))
    for columns in (400, 1, 156, 157, 400, 155):  # 100, 40,000, 257, 255, 100, 259 cells to a bucket
        cells = rods(4.0 * (k % columns) - 2.0 * columns, 4.0 * (k // columns) + 0.5, np.zeros(n), rng)
        g.set_cells(cells)
        for _ in range(2):
            g.step()
            got, o = g.get_cells(), np.argsort(cells["x"], kind="stable")
            np.testing.assert_array_equal(got["x"], cells["x"][o])
            np.testing.assert_array_equal(got["y"], cells["y"][o])
