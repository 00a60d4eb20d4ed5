"""Which form of the BBPGD solver runs, and its values against the traced solve
(always the streaming kernels) where the on-chip kernels are at their limits:
knots of cells whose entries find no room in their block's shared memory, in
the cluster and in the grid form, and sets beyond the on-chip kernels, which
the untraced streaming kernels take.

The form shows in the launches of a solve with one detection: the streaming
kernels need the mobilities and, for a planar colony, three packed arrays; the
on-chip kernels none of these, the planar ones the entries in order instead.
tests/test_host_programs.py checks that these colonies take the named forms
and leave that many groups without room."""
from __future__ import annotations

import numpy as np
import pytest

from pcc_b200 import abi, synth
from pcc_b200.device import Colony
from uneven import UNEVEN, uneven

pytestmark = pytest.mark.gpu

FORMS = [dict(precision=abi.PRECISION_FP64), dict(precision=abi.PRECISION_MIXED),
         dict(solver_variant=abi.SOLVER_GENERAL)]


def solve(cells: dict, trace_dir, trace: int, over: dict, tolerance: float):
    """One detection and its solve; the state it leaves and its launches."""
    p = abi.default_params(dt=3e-4, fixed_dt=1, tolerance=tolerance, max_recursive_iterations=1, log_bbpgd_trace=trace,
                           ghost_mode=abi.GHOSTS_NONE, **over)
    g = Colony(p)
    g.set_trace_dir(str(trace_dir))
    g.set_cells(cells)
    g.profiling(True)
    before = g.launches
    with pytest.raises(RuntimeError, match="Maximum number of constraint iterations"):
        g.solve(p.dt, 1)
    launches, iterations = g.launches - before, g.profile()["bbpgd_iterations"]
    return launches, iterations, g.get_cells(), g.constraints()


def compare(cells: dict, trace_dir, over: dict, on_chip: bool, tolerance: float = 5e-2):
    a, b = solve(cells, trace_dir, 0, over, tolerance), solve(cells, trace_dir, 2, over, tolerance)
    fewer = (1 if "solver_variant" in over else 3) if on_chip else 0
    assert b[0] - a[0] == fewer
    assert a[1] == b[1] > 10
    for k in a[2]:
        np.testing.assert_array_equal(a[2][k], b[2][k], err_msg=k)
    for k in ("gid_i", "gid_j", "gamma", "sd"):
        np.testing.assert_array_equal(a[3][k], b[3][k], err_msg=k)


@pytest.mark.parametrize("form", [0, 1, 2], ids=["fp64", "mixed", "3d"])
@pytest.mark.parametrize("size,forms", UNEVEN, ids=["-".join(map(str, s)) for s, _ in UNEVEN])
def test_uneven_colonies_bit_identical_to_streaming(size, forms, form, tmp_path):
    """The knots have no solution (BBPGD's residual stays above 0.9 for as long
    as it runs, from 0.5 at the start): the solve ends at the first residual
    under 2, some tens of iterations on."""
    compare(uneven(*size), tmp_path, FORMS[form], forms[form][0] != "streaming", tolerance=2.0)


@pytest.mark.parametrize("radius,form,on_chip", [(85.0, 0, True), (85.0, 2, False), (110.0, 0, False),
                                                 (110.0, 1, True), (150.0, 0, False), (150.0, 1, False)])
def test_largest_on_chip_and_smallest_streaming_sets(radius, form, on_chip, tmp_path):
    """65,056, 109,415 and 202,000 constraints."""
    cells = synth.dense_colony(radius, seed=1, lane_gap=0.0, end_gap=0.0)
    cells["x"], cells["y"] = cells["x"] * 0.985, cells["y"] * 0.985
    compare(cells, tmp_path, FORMS[form], on_chip)
