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
