"""What the host side does when memory is short, or another thread launches
meanwhile: its sources and objects over a CUDA runtime that only keeps books and
refuses what it is told to (tests/native).  No GPU is touched."""
import os
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "heronian-square-search_gb300" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"


def run_native(tmp_path, name, parts):
    exe = tmp_path / name
    built = subprocess.run(
        ["g++", "-std=c++17", "-O1", f"-I{CUDA}", "-o", str(exe), str(HERE / "native" / f"{name}.cpp"),
         *map(str, parts), "-pthread", "-Wl,--unresolved-symbols=ignore-all"],
        capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert ran.returncode == 0, ran.stdout + ran.stderr


@pytest.mark.parametrize("name", ["growth", "pressure", "open", "planner", "autotune"])
def test_host_side(tmp_path, name):
    run_native(tmp_path, name, [CSRC / "hss_plan.cpp", CSRC / "hss_prep.cpp"])


def test_launch_limits_of_two_threads(built, tmp_path):
    objects = CSRC.parent / "_build"
    run_native(tmp_path, "attributes", [objects / "hss_blocks.o", objects / "hss_kernels.o"])
