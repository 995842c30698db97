"""Bricks whose lists end at, before and after a batch of sweep records, and
sub-boxes of every width along x, against the oracle bit for bit, for volumes
of one and of two bundles."""

import warnings

import numpy as np
import pytest

LY1 = [(1.0, 0.004, 1.0, "r")]
LY2 = [(0.5, -0.004, 10.0, "p"), (1.0, 0.004, 1.0, "r")]


@pytest.mark.gpu
@pytest.mark.parametrize("bundles", [1, 2])
@pytest.mark.parametrize("n", [127, 128, 129, 256, 257, 513])
def test_lists_at_the_edge_of_a_batch(cuda, oracle_port, n, bundles):
    from fastpli_gb300.simulation import _Generator
    rng = np.random.default_rng(n + bundles)
    dim = (8, 8, 32)
    fibers = [[] for _ in range(bundles)]
    for i in range(n):  # one short segment each, in the one brick
        a = rng.uniform(0, 1, 3) * dim
        b = a + rng.normal(size=3) * [1.5, 1.5, 3.0]
        fibers[i % bundles].append(np.array([[*a, r := rng.uniform(0.1, 1.2)], [*b, r]]))
    layers = [LY2, LY1][:bundles]
    olab, ovec, _, _ = oracle_port.generate(dim, [0.0] * 3, 1.0, fibers, layers)
    assert (olab > 0).any()
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(fibers, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, _ = g.run_generation_device()
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
