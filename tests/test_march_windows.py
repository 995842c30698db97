"""The cooperative march against the oracle where its windows can go wrong:
step counts around a window's length, more labels than its table holds, steps
whose interpolated axis is zero (they must not attenuate), axes that are not
normalised, windows in which every step is birefringent, images that end inside
a ray tile.  Bound: the march's 1e-4 relative per pixel."""

import warnings

import numpy as np
import pytest


def _volume(dim, n_labels, zeros, seed):
    rng = np.random.default_rng(seed)
    coarse = rng.integers(0, n_labels, [-(-d // 3) for d in dim])
    label = np.kron(coarse, np.ones((3, 3, 3), np.int64))[:dim[0], :dim[1], :dim[2]]
    vec = rng.normal(size=dim + (3,))
    vec /= np.linalg.norm(vec, axis=-1, keepdims=True)
    vec[..., 2] = np.abs(vec[..., 2])
    vec[np.isin(label, np.arange(1, n_labels, 5))] *= zeros
    props = np.c_[rng.uniform(-0.004, 0.004, n_labels), rng.uniform(0, 20, n_labels)]
    props[::3, 0] = 0.0
    props[0] = (0.0, 1.5)
    if n_labels < 4:  # every step birefringent but outside
        label = np.maximum(label, 1)
        props[1:, 0] = 0.003
    return label.astype(np.int32), vec.astype(np.float32), props


@pytest.mark.gpu
@pytest.mark.parametrize("interpolate", ["Lerp", "Slerp"])
@pytest.mark.parametrize("dim,n_labels,zeros,flip", [
    ((19, 37, 1), 5, 1.0, False), ((9, 33, 7), 63, 0.0, False), ((12, 31, 8), 64, 0.0, True),
    ((21, 40, 9), 65, 0.0, False), ((6, 65, 17), 150, 1.5, False), ((17, 20, 33), 3, 1.0, True)])
def test_windows_match_oracle(cuda, oracle_port, interpolate, dim, n_labels, zeros, flip):
    from fastpli_gb300.simulation import _Simulator
    label, vec, props = _volume(dim, n_labels, zeros, sum(dim) + n_labels)
    kw = dict(step_size=1.0, light_intensity=26000.0, voxel_size=1.0, wavelength=525.0,
              tissue_refrection=1.0, interpolate=interpolate, untilt_sensor_view=True,
              flip_z=flip, filter_rotations=np.deg2rad(np.arange(0, 180, 20)))
    sim = _Simulator()
    sim.set_pli_setup(*kw.values())
    dev = [cuda.from_numpy(a).cuda() for a in (label, vec)]
    for theta, phi in np.deg2rad([(5.5, 0), (8.0, 133.0), (5.5, 270.0)]):
        ref, warn = oracle_port.simulate(label, vec, props, theta, phi, **kw)
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            img = sim.run_simulation_device(dim, *dev, props, theta, phi).cpu().numpy()
        assert (np.abs(img - ref) <= 1e-4 * np.abs(ref)).all()
