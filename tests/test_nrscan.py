"""The FP32 bounds on the Newton exit time's convergence measure
(csrc/nrscan.cuh): the host build of the header against the FP64 evaluation,
which must lie within them wherever there are bounds; contracted multiply-adds
and separate ones."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("contract", ["off", "fast"])
def test_bounds_hold_the_evaluation(tmp_path, contract):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "nrscan_check"
    subprocess.run([cxx, "-O2", "-std=c++17", f"-ffp-contract={contract}", "-I",
                    str(ROOT / "modpath-rw_gb300" / "csrc"), str(ROOT / "tests" / "nrscan_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, with_bounds, tried = r.stdout.split()
    assert ok == "ok" and int(with_bounds) > 2_000_000 and int(tried) == 4_000_000
