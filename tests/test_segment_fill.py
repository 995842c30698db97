"""Segment tables that the device fills from the points, against the oracle bit
for bit: on either side of the size up to which the host fills them, and for
fibers most of whose points lie outside the volume (more points than the
workspace has room for: the host fills the table after all)."""

import warnings

import numpy as np
import pytest

LY1 = [(1.0, 0.004, 1.0, "r")]
LY3 = [(0.333, -0.004, 10.0, "p"), (0.666, 0.0, 5.0, "b"), (1.0, 0.004, 1.0, "r")]
DIM, ORIGIN, VOXEL = (37, 41, 35), [-3.25, 1.5, 0.125], 0.7


def _walk(rng, n, outside):
    """n segments whose boxes reach into the volume; `outside` points beyond it
    at either end of the fiber."""
    lo = np.array(ORIGIN) + 1
    hi = lo + VOXEL * np.array(DIM) - 2
    pts = [rng.uniform(lo, hi)]
    while len(pts) < n + 1:
        step = rng.normal(size=3)
        q = pts[-1] + 0.6 * step / np.linalg.norm(step)
        if ((q > lo) & (q < hi)).all():
            pts.append(q)
    pts = np.column_stack([pts, rng.uniform(0.4, 2.2, n + 1)])
    if not outside:
        return pts
    far = np.tile([500.0, 600.0, 700.0, 1.0], (outside, 1))
    far[:, :3] += rng.uniform(-50, 50, (outside, 3))
    return np.concatenate([far, pts, far])


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,outside", [((1024,), 0), ((1025,), 0), ((700, 900, 401), 0),
                                           ((1100, 300), 40000)])
def test_filled_table_matches_oracle(cuda, oracle_port, sizes, outside):
    from fastpli_gb300.simulation import _Generator
    rng = np.random.default_rng(sum(sizes) + outside)
    fibers = [[_walk(rng, n, outside), _walk(rng, 1, 0)] for n in sizes]
    if len(sizes) == 1:
        fibers = [fibers[0][:1]]
    layers = [LY3, LY1, LY3][:len(sizes)]
    olab, ovec, oprop, _ = oracle_port.generate(DIM, ORIGIN, VOXEL, fibers, layers)
    assert (olab > 0).any()
    g = _Generator()
    g.set_volume(DIM, ORIGIN, VOXEL)
    g.set_fiber_bundles(fibers, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, prop, _ = g.run_generation_device()
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert np.array_equal(prop, oprop)
