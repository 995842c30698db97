"""The optic stage's map on images of few columns (a CTA shared by groups of
outputs, on both sides of 128 columns) and on axes so long that their weights
are kept part by part (70,000 outputs of 481 taps), against the oracle.  Bound,
for positive images: per axis and side n roundings in the sum that normalises
the taps and n in the sum of the products, n = 2 radius + block + 1 and 8 for
the exponentials, quotients and the block's mean: 8 (n + 8) 2^-53 relative."""

import numpy as np
import pytest

CASES = [((900, 1, 9), 20.0, 1.0), ((700, 1, 1), 3.0, 0.6), ((301, 14, 9), 5.0, 0.6),
         ((205, 127, 1), 0.71, 0.3), ((205, 128, 1), 0.71, 0.3), ((90, 43, 3), 0.5, 1.4),
         ((1, 600, 7), 9.0, 0.9), ((333, 129, 2), 0.0, 0.37), ((70000, 1, 1), 60.0, 1.0),
         ((1, 70000, 2), 60.0, 1.0)]


def _bound(sigma, scale):
    n = 2 * int(4 * sigma / scale + 0.5) + 1 / scale + 2
    return 8 * (n + 8) * 2.0 ** -53


@pytest.mark.gpu
@pytest.mark.parametrize("shape,sigma,scale", CASES)
def test_few_columns_match_oracle(cuda, shape, sigma, scale):
    from fastpli_gb300 import optic
    from oracle import optic as O
    img = np.random.default_rng(sum(shape)).uniform(1.0, 9000.0, shape)
    ref = O.filter_resample(img, sigma, scale)
    got = optic.filter_resample_device(cuda.from_numpy(img).cuda(), sigma, scale).cpu().numpy()
    assert got.shape == ref.shape
    nan = np.isnan(ref)
    assert np.array_equal(nan, np.isnan(got))
    assert (np.abs(got - ref)[~nan] <= _bound(sigma, scale) * ref[~nan]).all()
