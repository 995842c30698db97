"""The error bounds of the voxelizer's two-float fast path on the CPU: they are
what the roundings add up to at their worst, some 30 of them, so random draws,
whose roundings cancel for the greater part, must stay below a quarter of them."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "voxel_bound_check.cu")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("ucheck") / "ucheck")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), SRC, "-o", exe],
                   check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("length", ["1e-3", "1", "10", "1e3", "1e5"])
def test_errors_stay_well_inside_the_bounds(program, length):
    r = subprocess.run([program, "3", length, "400000", "0.25"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
