"""A host thread that marches page-locked volumes (uploads in slabs, launches on
streams of its own) beside one that runs tilting series on the device, and more
of them than stream sets are kept: every result is the one of the call alone."""

import threading
import warnings

import numpy as np
import pytest

from fastpli_gb300 import synth
from fastpli_gb300.simulation import _Generator, _Simulator

TILTS = [(np.deg2rad(5.5), k * np.pi / 2) for k in range(4)]


def _setup(seed, dim, n):
    w = synth.crossing(seed=seed, n_per_bundle=n, dim=dim, n_points=12)
    g = _Generator()
    g.set_volume(w.dim, w.origin, w.voxel_size)
    g.set_fiber_bundles(w.bundles, w.layers)
    s = _Simulator()
    s.set_pli_setup(1.0, 26000.0, w.voxel_size, 525.0, 1.0, "Slerp", True, False,
                    np.deg2rad([0.0, 30.0, 60.0, 90.0, 120.0, 150.0]))
    return w, g, s


@pytest.mark.gpu
@pytest.mark.parametrize("hosts", [1, 6])
def test_host_marches_beside_device_series(cuda, hosts):
    torch = cuda
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        wb, gb, sb = _setup(7, (200, 180, 96), 60)
        hl, hv, hp = gb.run_generation()  # page-locked
        ws, gs, ss = _setup(8, (48, 52, 32), 20)
        dl, dv, dp, _ = gs.run_generation_device()
        ref_host = [sb.run_simulation(wb.dim, hl, hv, hp, t, p).copy() for t, p in TILTS]
        ref_dev = [x.clone() for x in ss.run_tilts_device(ws.dim, dl, dv, dp, TILTS)]
    torch.cuda.synchronize()
    assert torch.from_numpy(hl).is_pinned()
    errors, left = [], [hosts]

    def host():
        try:
            s = _setup(7, (200, 180, 96), 60)[2]
            for _ in range(3):
                for k, (t, p) in enumerate(TILTS):
                    if not np.array_equal(s.run_simulation(wb.dim, hl, hv, hp, t, p), ref_host[k]):
                        errors.append(f"host march {k}")
        except Exception as e:
            errors.append(repr(e))
        left[0] -= 1

    def device():
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                while left[0] > 0:
                    out = ss.run_tilts_device(ws.dim, dl, dv, dp, TILTS, stream=stream)
                    stream.synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(out, ref_dev)):
                        errors.append("device series")
        except Exception as e:
            errors.append(repr(e))

    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        threads = [threading.Thread(target=host) for _ in range(hosts)]
        threads.append(threading.Thread(target=device))
        for t in threads:
            t.start()
        for t in threads:
            t.join(120)
    assert not any(t.is_alive() for t in threads)
    assert not errors, errors[:4]
