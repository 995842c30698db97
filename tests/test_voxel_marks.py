"""The voxelizer's sweep and its marked voxels against the oracle: labels,
vectors and the overlap warning bit for bit, on inputs that reach each of its
branches — lists of more than 256 segments (wider slots), bricks with few and
with many marked voxels (list and second sweep), exact ties, changing radii
(no certain layer), bricks without segments, volumes cut inside a brick."""

import warnings

import numpy as np
import pytest

LY1 = [(1.0, 0.004, 1.0, "r")]
LY3 = [(0.333, -0.004, 10.0, "p"), (0.666, 0.0, 5.0, "b"), (1.0, 0.004, 1.0, "r")]


def _curve(rng, size, n, r, bend=0.3, step=1.0, taper=0.0):
    p = rng.uniform(0, 1, 3) * size
    d = rng.normal(size=3)
    pts = []
    for _ in range(n):
        d = d / np.linalg.norm(d) + bend * rng.normal(size=3)
        p = p + step * d / np.linalg.norm(d)
        pts.append([*p, r * (1 + taper * rng.uniform(-1, 1))])
    return np.array(pts)


def _inputs(name):
    rng = np.random.default_rng(sum(map(ord, name)))
    dim, layers = (40, 33, 45), [LY3]
    size = np.array(dim, float)
    if name == "short":  # over 256 segments and many joints in a brick
        fibers = [[_curve(rng, size, 120, 3.0, step=0.4) for _ in range(40)]]
    elif name == "bent":  # wedges of voxels at equal distance from a joint
        fibers = [[_curve(rng, size, 12, 4.0, bend=0.8, step=5.0) for _ in range(12)]]
    elif name == "twice":  # every voxel tied with a later copy
        one = [_curve(rng, size, 8, 3.0, step=6.0) for _ in range(10)]
        fibers = [one + [f.copy() for f in one]]
    elif name == "taper":
        fibers = [[_curve(rng, size, 10, 3.0, step=5.0, taper=0.5) for _ in range(25)]]
    elif name == "bundles":  # a later bundle over an earlier one
        fibers = [[_curve(rng, size, 9, 2.5, step=5.0) for _ in range(8)] for _ in range(3)]
        layers = [LY3, LY1, LY3]
    elif name == "apart":  # two bundles that do not touch: no warning
        fibers = [[np.array([[5.0, 5, -3, 2], [5, 5, 50, 2]])],
                  [np.array([[30.0, 25, -3, 2], [30, 25, 50, 2]])]]
        layers = [LY1, LY3]
    elif name == "sparse":  # most bricks empty, a long and a degenerate segment
        dim = (70, 41, 67)
        fibers = [[np.array([[-200.0, -90, -150, 2], [260, 120, 190, 2]]),
                   np.array([[20.0, 20, 20, 1.5], [20, 20, 20, 1.5], [21, 20, 20, 1.5]])]]
    else:  # one fiber over everything
        fibers = [[np.array([[-40.0, 10, 20, 60], [90, 20, 25, 60]])]]
    return dim, fibers, layers


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["short", "bent", "twice", "taper", "bundles", "apart",
                                  "sparse", "wide"])
def test_marked_voxels_match_oracle(cuda, oracle_port, name):
    from fastpli_gb300.simulation import _Generator
    dim, fibers, layers = _inputs(name)
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(fibers, layers)
    olab, ovec, _, owarn = oracle_port.generate(dim, [0.0] * 3, 1.0, fibers, layers)
    assert (olab > 0).any()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, w = g.run_generation_device()
        only, _, _, _ = g.run_generation_device(only_label=True)
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert np.array_equal(only.cpu().numpy(), olab)
    if name in ("apart", "short", "twice"):  # one bundle, or bundles that do not touch
        assert w["overlap"] == owarn["overlap"] == 0
    if name == "bundles":
        assert w["overlap"] == 1
