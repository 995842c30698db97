"""Bricks with more marked voxels than a record holds, which a CTA resolves by
halves, against the oracle bit for bit with the overlap warning: fibers that
share their course with another (in one bundle and in two), radii that change,
8 segments and fewer (no records at all), as many marks per brick as records
hold but no room for them, lists longer than a batch, halves without voxels,
host buffers, and a batch."""

import warnings

import numpy as np
import pytest

LY1 = [(1.0, 0.004, 1.0, "r")]
LY3 = [(0.333, -0.004, 10.0, "p"), (0.666, 0.0, 5.0, "b"), (1.0, 0.004, 1.0, "r")]


def _walk(rng, size, n, r, taper=0.0):
    a, b = rng.uniform(-0.1, 1.1, (2, 3)) * size
    p = a + (b - a) * np.linspace(0, 1, n)[:, None]
    if n > 2:
        p += 0.6 * rng.normal(size=(n, 3))
    return np.column_stack([p, r * (1 + taper * rng.uniform(-1, 1, n))])


def _inputs(name, dim):
    rng = np.random.default_rng(sum(map(ord, name)) + sum(dim))
    size = np.array(dim, float)
    layers = [LY3]
    if name in ("twice", "twobundles"):
        one = [_walk(rng, size, 10, rng.uniform(1.5, 4)) for _ in range(16)]
        sets = [one, [f.copy() for f in one]] if name == "twobundles" else [one + one]
    elif name == "taper":
        sets = [[_walk(rng, size, 8, 4.0, 0.5) for _ in range(12)] for _ in range(2)]
    elif name == "few":  # 8 segments
        one = [_walk(rng, size, 2, 6.0) for _ in range(4)]
        sets = [one + one]
    elif name == "room":  # 34 segments: 104 entries for some 30 marks in each brick
        one = [_walk(rng, size, 18, 7.0)]
        sets = [one + [_walk(rng, size, 18, 7.0)]]
    else:  # "long list"
        one = [_walk(rng, size, 40, 2.0) for _ in range(20)]
        sets = [one, one]
    return sets, (layers + [LY1])[:len(sets)]


NAMES = ["twice", "twobundles", "taper", "few", "room", "long list"]


@pytest.mark.gpu
@pytest.mark.parametrize("dim", [(21, 30, 40), (66, 60, 70), (140, 161, 100)])
@pytest.mark.parametrize("name", NAMES)
def test_full_bricks_match_oracle(cuda, oracle_port, name, dim):
    from fastpli_gb300.simulation import _Generator
    sets, layers = _inputs(name, dim)
    olab, ovec, _, owarn = oracle_port.generate(dim, [0.0] * 3, 1.0, sets, layers)
    assert (olab > 0).any()
    g = _Generator()
    g.set_volume(dim, [0.0] * 3, 1.0)
    g.set_fiber_bundles(sets, layers)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        label, vector, _, w = g.run_generation_device()
        only, _, _, _ = g.run_generation_device(only_label=True)
        hlab, hvec, _ = g.run_generation()
        # the least workspace: records' space by segments only, or none
        least = cuda.empty(g.workspace_size(), dtype=cuda.uint8, device="cuda")
        llab, lvec, _, lw = g.run_generation_device(workspace=least)
    assert np.array_equal(label.cpu().numpy(), olab)
    assert np.array_equal(vector.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert np.array_equal(only.cpu().numpy(), olab)
    assert np.array_equal(hlab, olab) and np.array_equal(hvec.view(np.uint32),
                                                         ovec.view(np.uint32))
    assert np.array_equal(llab.cpu().numpy(), olab)
    assert np.array_equal(lvec.cpu().numpy().view(np.uint32), ovec.view(np.uint32))
    assert w["overlap"] == lw["overlap"] == owarn["overlap"]


@pytest.mark.gpu
def test_full_bricks_of_a_batch_match_oracle(cuda, oracle_port):
    from types import SimpleNamespace
    from fastpli_gb300.batch import TileBatch
    dims = [(21, 30, 40), (50, 33, 45)]
    tiles = []
    for dim, name in zip(dims, ("twobundles", "taper")):
        sets, layers = _inputs(name, dim)
        if name == "taper":  # a fiber longer than the volume beside them
            sets[0].append(np.array([[-80.0, -70, -90, 3], [120, 100, 130, 3]]))
        tiles.append(SimpleNamespace(dim=dim, origin=[0.0] * 3, voxel_size=1.0, bundles=sets,
                                     layers=layers, tilts=[(0.0, 0.0)]))
    setup = dict(light_intensity=26000.0, voxel_size=1.0, wavelength=525.0,
                 filter_rotations=np.deg2rad([0.0, 30, 60, 90, 120, 150]))
    batch = TileBatch(tiles, setup).allocate()
    batch.run()
    batch.capture()
    batch.replay()
    cuda.cuda.synchronize()
    for t, tile in enumerate(tiles):
        olab, ovec, _, _ = oracle_port.generate(tile.dim, [0.0] * 3, 1.0, tile.bundles,
                                                tile.layers)
        assert np.array_equal(batch.label(t).cpu().numpy(), olab)
        assert np.array_equal(batch.vector(t).cpu().numpy().view(np.uint32),
                              ovec.view(np.uint32))
