"""bench.py's reference arm where the reference's build is missing: one line
that says so, and no error."""
from __future__ import annotations

import json
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import sys
from pathlib import Path
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import bench, oracles
oracles.REF_DIR = Path({empty!r})
sys.argv = ["bench.py", "--impl", "reference", "--steps", "2", "--warmup", "1"]
bench.main()
"""


def test_reference_arm_says_unavailable(tmp_path):
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=str(ROOT), empty=str(tmp_path))],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and "\n" not in line["unavailable"] and set(line) == {"impl", "unavailable"}
