"""CPU tests of the CUDA-core TSMTTSM: the plan asks for the shared memory and the workspace that the kernel
touches, for all type pairs, Gram or not, widths up to 1000 (tests/cpp/plan_driver.cu); the row-streaming
kernel reads nothing behind a row (tests/cpp/rows_driver.cu)."""
import os
import subprocess

import pytest

from skinny_matmul_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_driver(tmp_path, name):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc is missing")
    exe = str(tmp_path / name)
    r = subprocess.run([nvcc] + build.ARCH + ["-O1", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                        "-I" + build.CSRC, os.path.join(ROOT, "tests", "cpp", name + ".cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout + r.stderr)
    return r.stdout


def test_plan_covers_every_group_of_cells(tmp_path):
    assert int(run_driver(tmp_path, "plan_driver").split()[1]) > 10**6


def test_rows_are_not_read_past_their_end(tmp_path):
    run_driver(tmp_path, "rows_driver")
