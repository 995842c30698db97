"""ROFL on either side of the map sizes at which the lanes of a pixel change,
more than 10 rotations among them, unmasked and with masks that leave the pixels
on the other side, none or one: the same fits bit for bit as a small map's."""

import warnings

import numpy as np
import pytest

from test_rofl import TAU, gold


@pytest.mark.gpu
@pytest.mark.parametrize("rot,pixels", [(12, 11999), (12, 12000), (18, 17999), (18, 18001)])
def test_lanes_on_either_side_of_the_rule(cuda, rot, pixels):
    from fastpli_gb300 import analysis
    name = "noisy6" if rot == 12 else "noisy9"
    data = gold()[name + "|in"]  # [pixels, 5, rotations]
    data = np.concatenate([data] * (rot // data.shape[2]), axis=2)[:53]

    def fit(n):
        d = data[np.arange(n) % len(data)].transpose(1, 0, 2)[:, :, None, :]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            out = analysis.rofl_device(cuda.from_numpy(np.ascontiguousarray(d)).cuda(), TAU, 3, 0)
        return out[:, 0].cpu().numpy()

    ref = fit(len(data))
    assert np.isfinite(ref).all()
    assert np.array_equal(fit(pixels), ref[np.arange(pixels) % len(data)])


@pytest.mark.gpu
@pytest.mark.parametrize("name,copies,pixels,left", [
    ("noisy9", 1, 1300, 1216), ("noisy9", 1, 1300, 1217), ("noisy9", 1, 80500, 79999),
    ("noisy9", 1, 80500, 80000), ("noisy9", 2, 18300, 17999), ("noisy9", 2, 18300, 18000),
    ("noisy6", 1, 90000, 40), ("noisy6", 2, 12400, 1), ("noisy9", 1, 700, 0)])
def test_masked_pixels_do_not_count(cuda, name, copies, pixels, left):
    from fastpli_gb300 import analysis
    data = gold()[name + "|in"]
    data = np.concatenate([data] * copies, axis=2)[:41]
    mask = np.zeros(pixels, bool)
    mask[np.random.default_rng(pixels + left).permutation(pixels)[:left]] = True

    def fit(n, m):
        d = data[np.arange(n) % len(data)].transpose(1, 0, 2)[:, :, None, :]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            out = analysis.rofl_device(cuda.from_numpy(np.ascontiguousarray(d)).cuda(), TAU, 3, 0,
                                       mask=None if m is None else m[:, None])
        return out[:, 0].cpu().numpy()

    ref = fit(len(data), None)
    got = fit(pixels, mask)
    assert np.isnan(got[~mask]).all()
    assert np.array_equal(got[mask], ref[np.arange(pixels) % len(data)][mask])
