"""The tile plans of the few-right-hand-side sweeps (rows_plan.cpp), executed on
the host as the kernel reads them (tests/rows_check.cpp): carriers and Poisson
factors at degrees 1 and 2, both Poisson pairings, ragged and graded meshes, for
both vector widths and several right-hand-side counts."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "pecs_gb300" / "csrc"


def test_row_plans(tmp_path):
    exe = tmp_path / "rows_check"
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", f"-I{CSRC}",
                        str(ROOT / "tests" / "rows_check.cpp"),
                        *[str(CSRC / f) for f in ("rows_plan.cpp", "mf.cpp", "dense.cpp", "problem.cpp")],
                        "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(out.stdout)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("OK")
