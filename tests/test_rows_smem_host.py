"""Shared memory of the few-right-hand-side sweeps' launches (rows_smem in
rows_plan.cpp), checked on the host (tests/rows_smem_check.cpp): levels that mix one
wide front with many small nodes, every chunk of right-hand sides, both vector
widths, level and flow launches."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "pecs_gb300" / "csrc"


def test_every_launch_fits(tmp_path):
    exe = tmp_path / "rows_smem_check"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", f"-I{CSRC}",
                        str(ROOT / "tests" / "rows_smem_check.cpp"),
                        *[str(CSRC / f) for f in ("rows_plan.cpp", "mf.cpp", "dense.cpp", "problem.cpp")],
                        "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(out.stdout)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("OK")
