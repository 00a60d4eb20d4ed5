"""bench.py's roofline figure: the bytes that an iteration cannot do without
over the measured copy rate, so a kernel that moved exactly those bytes at that
rate reads 1."""
from __future__ import annotations

import pytest

import bench


@pytest.mark.parametrize("precision,width", [("fp64", 8), ("mixed", 4)])
@pytest.mark.parametrize("phases", [[921_575], [900_000, 1_800_000, 2_700_000]])
def test_distinct_bytes_at_the_copy_rate_read_one(precision, width, phases):
    n, peak = 302_180, 6502.5
    constraint = 2 * 4 + 6 * width + 8 + 2 * 16  # ids, D and L, Phi, (gamma, g) in and out
    entry = 4 * width + 8 + 4
    cell = 4 + 4 * width + 2 * 4 * width
    prof = {"bbpgd_iterations": 0, "bbpgd_algo_bytes": 0.0, "bbpgd_launches": len(phases), "solves": 2,
            "cell_solves": 2.0 * n}
    moved = 0.0
    for k, m in enumerate(phases):
        its = 100 * (k + 1)
        ac, an = (312, 288) if precision == "fp64" else (192, 144)
        prof["bbpgd_iterations"] += its
        prof["bbpgd_algo_bytes"] += its * (ac * m + an * n)
        moved += its * (m * (constraint + 2 * entry) + n * cell)
    prof["bbpgd_ms"] = moved / (peak * 1e9) * 1e3
    line = bench.roofline(prof, precision, {"hbm_gbs": peak})
    assert line["bound"] == "hbm" and abs(line["frac"] - 1.0) < 1e-12 and abs(line["achieved"] - peak) < 1e-8
