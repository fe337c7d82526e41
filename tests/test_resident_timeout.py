"""The bounded waits of the resident solves: with a limit of one poll they run
out, every block says so, the kernel ends by itself and the same buffers solve
the system afterwards.  (The context reports timed_out as FS_TIMEOUT.)"""
import os
import subprocess

import pytest

import fluid_simulator_backup_b200 as fs
from fluid_simulator_backup_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not os.path.exists(build.NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("resident") / "resident_timeout")
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-I" + build.CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "resident_timeout.cu"), "-o", exe, fs.LIB_PATH, "-Xlinker",
                    "-rpath," + os.path.dirname(fs.LIB_PATH)], check=True, timeout=300)
    return exe


def test_builds_against_the_library(program):
    assert os.access(program, os.X_OK)


@pytest.mark.gpu
def test_waits_that_run_out_are_reported(program):
    out = subprocess.run([program], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
    fp64, red_black = (tuple(map(int, line.split())) for line in out.stdout.splitlines())
    assert fp64[:3] == (1, 0, 1) and 20 < fp64[3] < 1000      # then converged (PCG_CONVERGED)
    assert red_black == (1, 0, 2, 20)                          # then at its cap (PCG_MAXITER)
