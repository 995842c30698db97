"""Segments longer than the volume, up to lengths whose squares overflow in
FP32 and FP64.  On the CPU a replay of the bricks' sweep (host build of the
kernel's functions): every voxel that it does not mark has the winner and layer
of the FP64 evaluation of all candidates.  On the GPU labels, vectors and
warnings against the oracle bit for bit, with short fibers in the same bricks."""

import os
import shutil
import subprocess
import warnings

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "voxel_brick_check.cu")
LENGTHS = ["1e3", "1e6", "1e9", "2e9", "1e12", "1e16", "1e19", "1.6e19", "1e20", "1e160"]
LY1 = [(1.0, 0.004, 1.0, "r")]
LY3 = [(0.333, -0.004, 10.0, "p"), (0.666, 0.0, 5.0, "b"), (1.0, 0.004, 1.0, "r")]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("bcheck") / "bcheck")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-fmad=false", "-Xcompiler",
                    "-ffp-contract=off,-fopenmp", "-I", os.path.join(ROOT, "include"), SRC,
                    "-o", exe], check=True, capture_output=True)
    return exe


def replay(program, *args):
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    words = [w for w in r.stdout.split() if not w.startswith("(")]
    return dict(zip(words[::2], words[1::2]))


@pytest.mark.parametrize("length", LENGTHS)
def test_unmarked_voxels_are_certain(program, length):
    replay(program, 9, 96, 80, 64, 3, 12, 2, 0, length)


@pytest.mark.parametrize("radius,points,taper", [(1e20, 3, 0), (4, 9, 0), (4, 9, 0.5)])
def test_unmarked_voxels_are_certain_at_other_radii(program, radius, points, taper):
    replay(program, 5, 61, 43, 50, radius, 14, points, taper, 0)


@pytest.mark.parametrize("args", [
    (1, 256, 128, 64, 5, 100, 2, 0, 0), (1, 512, 128, 64, 5, 100, 2, 0, 0),
    (1, 1024, 64, 64, 5, 50, 2, 0, 0), (1, 1024, 64, 64, 1.5, 500, 2, 0, 0),
    (1, 96, 80, 64, 3, 60, 2, 0, 66), (1, 96, 80, 64, 3, 60, 2, 0, 1e5)])
def test_few_close_calls_whatever_the_length(program, args):
    """A margin of at most 1.1e-6 (2 * 40)^2 = 0.007 either side of the layers
    at r^2 and 0.56 r^2: 4 * 0.007 / r^2 of a fiber's voxels, and as many where
    two fibers meet."""
    bound = 0.015 if args[4] > 2 else 0.03
    out = replay(program, *args)
    assert float(out["marked"]) <= bound * float(out["inside"]) and out["over"] == "0", out


@pytest.mark.gpu
@pytest.mark.parametrize("bundles,fibers", [(1, 20), (1, 300), (2, 260)])
def test_lists_of_two_point_fibers_match_oracle(cuda, oracle_port, bundles, fibers):
    """More long segments in a brick than it sweeps at a time, and few."""
    from fastpli_gb300.simulation import _Generator
    rng = np.random.default_rng(fibers)
    dim = (43, 37, 70)
    sets = []
    for _ in range(bundles):
        m = rng.uniform(0, 1, (fibers, 3)) * dim
        d = rng.normal(size=(fibers, 3))
        d *= 300 / np.linalg.norm(d, axis=1, keepdims=True)
        r = rng.uniform(1.0, 5.0, fibers)
        sets.append([np.column_stack([np.stack([a - v, a + v]), [q, q]])
                     for a, v, q in zip(m, d, r)])
    layers = [LY3, LY1][:bundles]
    olab, ovec, _, owarn = oracle_port.generate(dim, [0.0] * 3, 1.0, sets, layers)
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(sets, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, w = g.run_generation_device()
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert w["overlap"] == owarn["overlap"]


@pytest.mark.gpu
@pytest.mark.parametrize("length", LENGTHS)
def test_long_segments_match_oracle(cuda, oracle_port, length):
    from fastpli_gb300.simulation import _Generator
    rng = np.random.default_rng(11)
    dim = (48, 57, 40)
    long, short = [], []
    for _ in range(8):
        d = rng.normal(size=3)
        d = d / np.linalg.norm(d) * float(length)
        m, e = rng.uniform(0.2, 0.8, 3) * dim, rng.uniform(0.2, 0.8)
        long.append(np.array([[*(m - e * d), 3.0], [*(m + (1 - e) * d), 3.0]]))
        q = rng.uniform(0.1, 0.9, 3) * dim + np.linspace(-4, 4, 5)[:, None] * rng.normal(size=3)
        short.append(np.column_stack([q, np.full(5, 2.0)]))
    fibers, layers = [long, short], [LY3, LY1]
    with np.errstate(all="ignore"):
        olab, ovec, _, owarn = oracle_port.generate(dim, [0.0] * 3, 1.0, fibers, layers)
    assert (olab > 0).any()
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(fibers, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, w = g.run_generation_device()
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert w["overlap"] == owarn["overlap"]
