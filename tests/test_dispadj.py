"""The displacement's adjoint (csrc/dispadj.cuh) shares quotients between its
outputs; its rounding errors stay those of the formulas with every quotient
written out: within 2 %, the outputs of the gradient (velocity, correction and
dispersivities) each."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_rounding_errors_are_the_plain_quotients(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "dispadj_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "modpath-rw_gb300" / "csrc"),
                    str(ROOT / "tests" / "dispadj_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    ratios = [float(v) for v in r.stdout.split()]
    assert len(ratios) == 9 and max(ratios[:8]) < 1.02, ratios
