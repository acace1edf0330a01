"""CPU test: the plan of the CUDA-core TSMTTSM asks for the shared memory and the workspace that its
kernel touches, for all type pairs, Gram or not, widths up to 1000 (tests/cpp/plan_driver.cu)."""
import os
import subprocess

import pytest

from skinny_matmul_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plan_covers_every_group_of_cells(tmp_path):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc is missing")
    exe = str(tmp_path / "plan_driver")
    r = subprocess.run([nvcc] + build.ARCH + ["-O1", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                        "-I" + build.CSRC, os.path.join(ROOT, "tests", "cpp", "plan_driver.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[1]) > 10**6
