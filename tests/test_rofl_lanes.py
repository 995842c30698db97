"""ROFL with 16, 4 and 1 lanes per pixel (small, middle and large maps): the
same fits bit for bit, the maps being copies of the same pixels, with a last
warp that is not full and masked pixels among the others."""

import numpy as np
import pytest

from test_rofl import TAU, gold


@pytest.mark.gpu
@pytest.mark.parametrize("name,rot,grad", [("noisy6", 6, False), ("noisy9", 9, False),
                                           ("noisy9", 9, True), ("noisy9", 18, False)])
def test_lane_counts_agree(cuda, name, rot, grad):
    import warnings
    from fastpli_gb300 import analysis
    data = gold()[name + "|in"]  # [pixels, 5, rotations]
    data = np.concatenate([data] * (rot // data.shape[2]), axis=2)[:61]

    def fit(copies, masked=False):
        n = len(data) * copies
        d = np.tile(data, (copies, 1, 1)).transpose(1, 0, 2)[:, :, None, :]
        mask = np.ones((n, 1), bool)
        if masked:
            mask[::7] = False
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            out = analysis.rofl_device(cuda.from_numpy(np.ascontiguousarray(d)).cuda(), TAU, 3, 0,
                                       grad, mask=mask)
        return out[:, 0].cpu().numpy(), mask[:, 0]

    ref, _ = fit(1)
    assert np.isfinite(ref).all()
    for copies in (21, 1320):  # 1,281 and 80,520 pixels
        got, mask = fit(copies, masked=True)
        assert np.isnan(got[~mask]).all()
        assert np.array_equal(got[mask], np.tile(ref, (copies, 1))[mask])
