"""Host-side programs built by nvcc from the library's own sources and run on
the CPU, with stand-ins for the CUDA calls that would need a GPU."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not Path(NVCC).exists(), reason="nvcc not found")


def run(name: str, tmp_path, *args, stdin: str | None = None) -> str:
    """Builds tests/<name>.cu; what other sources of the library define and the program does not call stays unresolved."""
    exe = tmp_path / name
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-Xlinker",
                    "--unresolved-symbols=ignore-all", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'proliferatingcellcollectives-idp_b200' / 'csrc'}", str(ROOT / "tests" / f"{name}.cu"),
                    "-o", str(exe)], check=True, timeout=600)
    r = subprocess.run([str(exe), *args], input=stdin, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_contact_download_leaves_no_copy_in_flight(tmp_path):
    assert run("contact_download", tmp_path).startswith("ok")


def test_general_solver_grids_fit_each_kernel(tmp_path):
    assert run("solver_grids", tmp_path).startswith("ok")


def test_on_chip_solver_takes_the_forms_its_tests_name(tmp_path):
    """The dispatch and the room of every block for the colonies of
    tests/test_gpu_resident_forms.py, from the oracle's contact lists, and the
    kernel's bounds for sets of several detections one after another."""
    import numpy as np

    from oracles import OracleColony
    from pcc_b200 import abi, synth
    from uneven import UNEVEN, uneven

    def contacts(cells, tol=0.25):
        o = OracleColony(abi.default_params(ghost_mode=abi.GHOSTS_NONE))
        o.set_cells(cells)
        c = o.detect(tol, 0)
        i, j = np.minimum(c["gid_i"], c["gid_j"]), np.maximum(c["gid_i"], c["gid_j"])
        order = np.lexsort((j, i))
        return i[order], j[order]

    lines, want = [], []

    def ask(real, full, cells, lists, expect):
        i, j = np.concatenate([a for a, _ in lists]), np.concatenate([b for _, b in lists])
        pairs = " ".join(f"{a} {b}" for a, b in zip(i, j))
        lines.append(f"{real} {full} {len(lists)} {len(cells['x'])} {len(i)} {pairs}")
        want.append(expect)

    kinds = [("d", 0), ("f", 0), ("d", 1)]
    for size, forms in UNEVEN:
        cells = uneven(*size)
        found = contacts(cells)
        for (real, full), (form, without) in zip(kinds, forms):
            ask(real, full, cells, [found], (form, without))
    for radius, forms in [(9.0, ("cluster", "cluster", "cluster")), (27.0, ("grid", "cluster", "grid")),
                          (60.0, ("grid", "grid", "grid")), (85.0, ("grid", "grid", "streaming")),
                          (110.0, ("streaming", "grid", "streaming"))]:
        cells = synth.dense_colony(radius, seed=1, lane_gap=0.0, end_gap=0.0)
        cells["x"], cells["y"] = cells["x"] * 0.985, cells["y"] * 0.985
        found = contacts(cells)
        for (real, full), form in zip(kinds, forms):
            ask(real, full, cells, [found], (form, 0))
    # several detections: shrinking parts of the list again, from 1 cell up
    rng = np.random.default_rng(0)
    for radius in np.geomspace(2.0, 25.0, 40):
        cells = synth.dense_colony(float(radius), seed=int(100 * radius), lane_gap=0.0, end_gap=0.0)
        i, j = contacts(cells)
        lists = [(i, j)]
        for _ in range(int(rng.integers(0, 12))):
            keep = rng.random(len(i)) < rng.random()
            lists.append((i[keep], j[keep]))
        for real, full in kinds:
            ask(real, full, cells, lists, None)
    out = run("resident_shapes", tmp_path, stdin="\n".join(lines) + "\n").splitlines()
    assert len(out) == len(want)
    for got, expect in zip(out, want):
        form, _, without = got.split()
        assert expect is None or (form, int(without)) == expect, (got, expect)


def test_noalloc_scratch_is_the_current_contexts(tmp_path):
    assert run("noalloc_scratch", tmp_path).startswith("ok")
