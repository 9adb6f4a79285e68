"""Division and square root on the integer pipe (csrc/fpbits.cuh): the host
build of the header against the IEEE-754 operators, bit for bit, with the FP32
approximations that start the digits perturbed either way."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_div_and_sqrt_match_the_operators(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "divsqrt_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "modpath-rw_gb300" / "csrc"),
                    str(ROOT / "tests" / "fpbits_divsqrt_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok "), r.stdout
    assert int(r.stdout.split()[1]) > 5_000_000
