"""The optic stage's combined blur-and-resample map against the oracle at its
edges: lines shorter than the kernel (repeated reflection), more output than
input pixels (empty blocks), no blur, one angle, output counts around the rows a
thread takes together, non-finite pixels.  Bound: the longest sum has n <= 2 *
255 + 1 / scale + 1 terms per axis, each rounded to 2^-53: (n + 2) 2^-52 per
axis and as much for the oracle, below 1e-13 relative for positive images."""

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shape,sigma,scale", [
    ((5, 3, 2), 1.3, 0.5), ((1, 9, 1), 0.8, 0.6), ((2, 2, 9), 3.0, 0.5), ((33, 20, 6), 0.0, 0.3),
    ((7, 6, 3), 0.6, 1.7), ((64, 31, 9), 0.71, 0.2 / 1.33), ((41, 130, 1), 0.5, 0.25),
    ((20, 27, 3), 9.0, 0.15), ((129, 17, 4), 0.7, 1.0)])
def test_map_matches_oracle(cuda, shape, sigma, scale):
    from fastpli_gb300 import optic
    from oracle import optic as O
    img = np.random.default_rng(sum(shape)).uniform(1.0, 9000.0, shape)
    ref = O.filter_resample(img, sigma, scale)
    got = optic.filter_resample_device(cuda.from_numpy(img).cuda(), sigma, scale).cpu().numpy()
    assert got.shape == ref.shape
    nan = np.isnan(ref)
    assert np.array_equal(nan, np.isnan(got))
    assert (np.abs(got - ref)[~nan] <= 1e-13 * np.abs(ref[~nan])).all()


@pytest.mark.gpu
def test_map_spreads_non_finite_pixels_as_the_filter(cuda):
    from fastpli_gb300 import optic
    from oracle import optic as O
    img = np.random.default_rng(3).uniform(1.0, 9000.0, (40, 36, 2))
    img[7, 9, 0], img[20, 30, 1] = np.inf, np.nan
    ref = O.filter_resample(img, 0.71, 0.5)
    got = optic.filter_resample_device(cuda.from_numpy(img).cuda(), 0.71, 0.5).cpu().numpy()
    for kind in (np.isnan, np.isposinf):
        assert np.array_equal(kind(ref), kind(got))
