"""The reciprocals, square roots, conversions and comparisons that the kernels use
in place of FP64-pipe instructions, and the training sigmoid, hold their stated
bounds on the device: tests/cxx/fp64_check.cu, built with nvcc and run."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_stated_bounds(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fp64_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3",
                    "-I", os.path.join(REPO, "include"), "-I", os.path.join(REPO, "persiansph_gb300", "csrc"),
                    os.path.join(REPO, "tests", "cxx", "fp64_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(res.stdout)
    assert res.returncode == 0 and "failures 0" in res.stdout, res.stdout + res.stderr
