"""What the host side does when memory is short: the C ABI's source over a CUDA
runtime that only records allocations and refuses those it is told to
(tests/native).  No GPU is touched."""
import os
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "heronian-square-search_gb300" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"


def run_native(tmp_path, name):
    exe = tmp_path / name
    built = subprocess.run(
        ["g++", "-std=c++17", "-O1", f"-I{CUDA}", "-o", str(exe), str(HERE / "native" / f"{name}.cpp"),
         str(CSRC / "hss_plan.cpp"), str(CSRC / "hss_prep.cpp"), "-pthread", "-Wl,--unresolved-symbols=ignore-all"],
        capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert ran.returncode == 0, ran.stdout + ran.stderr


@pytest.mark.parametrize("name", ["growth", "pressure", "open", "planner"])
def test_host_side(tmp_path, name):
    run_native(tmp_path, name)
