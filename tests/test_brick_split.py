"""Volumes of few bricks, which several CTAs share, against the oracle bit for
bit: on both sides of each rule (bricks by 8, 4, 2 and 1 CTAs, marked voxels by
eights and by the record), x extents that leave a brick's last parts empty, and
bricks with more marked voxels than a record holds (every segment twice)."""

import warnings

import numpy as np
import pytest

LY1 = [(1.0, 0.004, 1.0, "r")]
LY3 = [(0.333, -0.004, 10.0, "p"), (0.666, 0.0, 5.0, "b"), (1.0, 0.004, 1.0, "r")]


@pytest.mark.gpu
@pytest.mark.parametrize("bundles,twice", [(1, False), (2, False), (1, True)])
@pytest.mark.parametrize("dim", [
    (3, 8, 32),     # 1 brick: 8 CTAs, five of them without voxels
    (15, 151, 20),  # 38 bricks: 8
    (17, 97, 25),   # 39: 4
    (29, 150, 31),  # 76: 4
    (50, 81, 13),   # 77: 2
    (64, 149, 32),  # 152: 2
    (70, 128, 40),  # 288: 1, marks by eights
    (127, 150, 99),  # 1,216: 1, marks by eights
    (128, 151, 97),  # 1,216: the same, cut elsewhere
    (136, 152, 97),  # 1,292: 1, whole records
])
def test_few_bricks_match_oracle(cuda, oracle_port, dim, bundles, twice):
    from fastpli_gb300.simulation import _Generator
    rng = np.random.default_rng(sum(dim) + bundles)
    size = np.array(dim, float)
    fibers = [[] for _ in range(bundles)]
    for i in range(24):
        a, b = rng.uniform(-0.1, 1.1, (2, 3)) * size
        t = np.linspace(0, 1, 14)[:, None]
        p = a + (b - a) * t + rng.normal(size=(14, 3))
        fibers[i % bundles].append(np.column_stack([p, np.full(14, rng.uniform(0.8, 3.0))]))
    if twice:
        fibers[0] += [f.copy() for f in fibers[0]]
    layers = [LY3, LY1][:bundles]
    olab, ovec, _, _ = oracle_port.generate(dim, [0.0] * 3, 1.0, fibers, layers)
    assert (olab > 0).any()
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(fibers, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, _ = g.run_generation_device()
        only, _, _, _ = g.run_generation_device(only_label=True)
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert np.array_equal(only.cpu().numpy(), olab)
