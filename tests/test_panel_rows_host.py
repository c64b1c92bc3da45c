"""The tile plans of FP64 banks with many right-hand sides (panel_plan.cpp), executed on
the host as the kernel reads them (tests/panel_rows_check.cpp)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "pecs_gb300" / "csrc"


def test_fp64_panel_plans(tmp_path):
    exe = tmp_path / "panel_rows_check"
    src = ("panel_plan.cpp", "rows_plan.cpp", "mf.cpp", "dense.cpp", "problem.cpp")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-pthread", f"-I{CSRC}",
                        str(ROOT / "tests" / "panel_rows_check.cpp"), *[str(CSRC / f) for f in src], "-o", str(exe)],
                       capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(out.stdout)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip().endswith("OK")
