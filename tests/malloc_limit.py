"""Runs a test's body in a process of its own with malloc_limit.cpp preloaded
(a device whose free memory the body sets)."""
import ctypes
import os
import shutil
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
_SO = "MPRW_TEST_MALLOC_LIMIT"


def limit():
    """The preloaded limit, within the body."""
    lib = ctypes.CDLL(os.environ[_SO])
    lib.malloc_limit_live.restype = ctypes.c_size_t
    lib.malloc_limit_refused.restype = ctypes.c_long
    lib.malloc_limit_set.argtypes = [ctypes.c_size_t]
    lib.malloc_limit_refuse.argtypes = [ctypes.c_long]
    return lib


def run(body: str, tmp_path) -> None:
    so = tmp_path / "malloc_limit.so"
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no C++ compiler"
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", "-std=c++17", str(ROOT / "tests" / "malloc_limit.cpp"), "-o",
                    str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=os.pathsep.join(
        [str(ROOT), str(ROOT / "modpath-rw_gb300"), str(ROOT / "tests")]))
    env[_SO] = str(so)
    r = subprocess.run([sys.executable, "-c", body], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, f"{r.returncode}\n{r.stdout}{r.stderr}"
