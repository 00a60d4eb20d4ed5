"""The on-chip BBPGD kernels (a cluster of 1 to 16 blocks, or the whole GPU)
against the streaming kernels, bit for bit.

`log_bbpgd_trace = 2` records every solve without changing it and always runs
the streaming kernels, so the same colony solved with and without it compares
the two.  The radii give constraint sets on both sides of every change of form:
none at all, one block (up to 512 constraints), clusters of 2 to 16 blocks,
the grid form, and sets that fit no shared memory; the crowded colony has a
cell whose entries outgrow a block's even share."""
from __future__ import annotations

import numpy as np
import pytest

from pcc_b200 import abi, synth
from pcc_b200.device import Colony

pytestmark = pytest.mark.gpu


def squeezed(radius: float, by: float, seed: int = 1) -> dict:
    """A dense packing drawn together, so that its cells overlap and BBPGD has work to do."""
    c = synth.dense_colony(radius, seed=seed, lane_gap=0.0, end_gap=0.0)
    c["x"], c["y"] = c["x"] * by, c["y"] * by
    return c


def solve(cells: dict, trace_dir, trace: int, **over):
    p = abi.default_params(dt=3e-4, fixed_dt=1, tolerance=2e-2, max_recursive_iterations=60, log_bbpgd_trace=trace,
                           **over)
    g = Colony(p)
    g.set_trace_dir(str(trace_dir))
    g.set_cells(cells)
    st = g.solve(p.dt, 1)
    return st, g.get_cells(), g.constraints()


def assert_same(a, b):
    assert a[0] == b[0]
    for k in a[1]:
        np.testing.assert_array_equal(a[1][k], b[1][k], err_msg=k)
    for k in ("gid_i", "gid_j", "gamma", "sd"):
        np.testing.assert_array_equal(a[2][k], b[2][k], err_msg=k)


FORMS = [dict(precision=abi.PRECISION_FP64), dict(precision=abi.PRECISION_MIXED),
         dict(solver_variant=abi.SOLVER_GENERAL)]


@pytest.mark.parametrize("over", FORMS, ids=["fp64", "mixed", "3d"])
@pytest.mark.parametrize("radius", [1.2, 3.0, 6.0, 9.0, 13.0, 18.0, 27.0, 60.0])
def test_on_chip_solve_bit_identical_to_streaming(radius, over, tmp_path):
    cells = squeezed(radius, 0.985)
    assert_same(solve(cells, tmp_path, 0, **over), solve(cells, tmp_path, 2, **over))


@pytest.mark.parametrize("radius", [120.0, 160.0])
@pytest.mark.parametrize("over", FORMS[:2], ids=["fp64", "mixed"])
def test_streaming_with_long_chunks_bit_identical_to_traced(over, radius, tmp_path):
    """Phases on both sides of 500,000 constraints, where the untraced
    streaming kernel changes from three to four blocks per SM."""
    cells = squeezed(radius, 0.985)
    a, b = solve(cells, tmp_path, 0, **over), solve(cells, tmp_path, 2, **over)
    assert 500_000 < a[0]["n_constraints"] < 1_212_416  # 592 chunks of up to 2,048
    assert_same(a, b)


@pytest.mark.parametrize("over", FORMS, ids=["fp64", "mixed", "3d"])
def test_one_cell_and_no_constraints(over, tmp_path):
    cells = {k: np.asarray(v, np.int32 if k == "age" else float) for k, v in abi.seed_cell(4).items()}
    a, b = solve(cells, tmp_path, 0, **over), solve(cells, tmp_path, 2, **over)
    assert a[0]["n_constraints"] == 0 and a[0]["bbpgd_iterations"] == 10
    assert_same(a, b)


@pytest.mark.parametrize("over", FORMS, ids=["fp64", "mixed", "3d"])
@pytest.mark.parametrize("around", [28, 400])
def test_crowded_cells(around, over, tmp_path):
    """Long cells laid across a row of others: entry counts from 1 to many, so
    the order of a block's cells by entry count and the padding are uneven."""
    n = around
    x = np.concatenate([np.arange(n) * 0.62, [0.3 * n * 0.62, 0.7 * n * 0.62]])
    y = np.concatenate([np.zeros(n), [1.1, -1.1]])
    th = np.concatenate([np.full(n, np.pi / 2) + 1e-3 * np.arange(n), [1e-3, 2e-3]])
    length = np.concatenate([np.linspace(1.0, 1.6, n), [1.99, 1.95]])
    cells = {"x": x, "y": y, "z": np.zeros(n + 2), "q0": np.cos(th / 2), "q1": np.zeros(n + 2),
             "q2": np.zeros(n + 2), "q3": np.sin(th / 2), "length": length, "l0": np.ones(n + 2),
             "diameter": np.full(n + 2, 0.5), "age": np.ones(n + 2, np.int32)}
    o = np.argsort(x, kind="stable")
    cells = {k: v[o] for k, v in cells.items()}
    assert_same(solve(cells, tmp_path, 0, **over), solve(cells, tmp_path, 2, **over))


def test_iteration_limit_is_an_error_in_both(tmp_path):
    """A solve that runs out of iterations raises the reference's message (what
    it leaves behind differs: the traced solve stores gamma at every iteration)."""
    cells = squeezed(9.0, 0.985)
    for trace in (0, 2):
        p = abi.default_params(dt=3e-4, fixed_dt=1, tolerance=1e-9, max_bbpgd_iterations=25, log_bbpgd_trace=trace)
        g = Colony(p)
        g.set_trace_dir(str(tmp_path))
        g.set_cells(cells)
        with pytest.raises(RuntimeError, match="BBPGD did not converge"):
            g.solve(p.dt, 1)
