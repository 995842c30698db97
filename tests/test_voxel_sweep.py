"""The bounds that let the voxelizer's one FP32 sweep name a voxel's segment, on
the CPU (host build of the same code) over every voxel of random segment boxes:
short, long and degenerate segments, thick ones and ones that taper."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "voxel_sweep_check.cu")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("scheck") / "scheck")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), SRC, "-o", exe],
                   check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("voxel,length,radius,fibers,taper", [
    (1, 5, 2, 60, 0), (1, 5, 2, 60, 1), (0.7, 300, 1.2, 20, 0), (0.1, 0.5, 0.3, 200, 1),
    (1, 1e5, 3, 12, 0), (1, 0.02, 4, 40, 1), (1, 0, 3, 10, 0)])
def test_bounds_hold(checker, voxel, length, radius, fibers, taper):
    r = subprocess.run([checker, "7", *map(str, (voxel, length, radius, fibers, taper))],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
