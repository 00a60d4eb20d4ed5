"""A colony created after the process has reset its own CUDA context solves as
one created before: nothing that belongs to a context outlives it."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import ctypes, sys
sys.path.insert(0, {root!r})
import pcc_pkg
pcc_pkg.load_package()
from pcc_b200 import abi, synth
from pcc_b200.device import Colony

forms = [dict(precision=abi.PRECISION_FP64), dict(precision=abi.PRECISION_MIXED),
         dict(solver_variant=abi.SOLVER_GENERAL)]

def solve(radius, over):
    p = abi.default_params(dt=3e-4, fixed_dt=1, **over)
    g = Colony(p)
    g.set_cells(synth.dense_colony(radius))
    st = g.solve(p.dt, 1)
    g.close()
    return st

before = [solve(r, f) for r in (9.0, 60.0) for f in forms]
cuda, dev = ctypes.CDLL("libcuda.so.1"), ctypes.c_int()
assert cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuDevicePrimaryCtxReset_v2(dev) == 0
assert [solve(r, f) for r in (9.0, 60.0) for f in forms] == before
"""


def test_solve_after_context_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=str(ROOT))], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
