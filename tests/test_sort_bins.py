"""The cell sort's bins and scan positions (persiansph_gb300/csrc/psph_bins.cuh)
stay exact up to 2^28 cells with four slabs a cell, 2^31 bins: the functions that
the kernels call, compiled for the host with nvcc, so it runs without a GPU."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bins_at_the_limit_of_cells(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "bins_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "persiansph_gb300", "csrc"),
                    os.path.join(REPO, "tests", "cxx", "bins_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    assert "mismatches 0" in res.stdout
