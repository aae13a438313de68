"""The Wolff bond test's exponential (marked gpu): tests/c/bond_exp.cu compares the decisions of xy_device.cuh with
CUDA's __expf for every FP32 argument."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bond_decisions_are_those_of_expf_for_every_argument(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not installed")
    exe = str(tmp_path / "bond_exp")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "slsf-rs_b200", "csrc"), os.path.join(ROOT, "tests", "c", "bond_exp.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "differences 0\n", r.stdout + r.stderr
