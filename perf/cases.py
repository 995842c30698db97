"""The framework's work, as cases whose time and results can be compared.

Each case is one thing a program does through the public entry points: the
voxelizer (``_Generator``), the ray march (``_Simulator``), a captured batch of
uneven tiles (``TileBatch``), the drop-in host API (``Simpli``), the optic
stage with its noise and epa, and ROFL.  Sizes are the repository's own
workloads (``fastpli_gb300.synth``) and ragged ones around them.

``listed`` gives the cases, ``draw`` more of the same ranges, ``prepare`` the
inputs and plans a program keeps, ``run`` one pass, ``work`` the bytes and
operations it cannot do without, and ``exact`` what it returns in 64 bits,
computed with plain torch.
"""

import math

import numpy as np
import torch

from fastpli_gb300 import analysis, optic, synth
from fastpli_gb300.batch import TileBatch
from fastpli_gb300.simpli import Simpli
from fastpli_gb300.simulation import _Generator, _Simulator

LAYERS_2 = [(0.75, 0.0, 10.0, "b"), (1.0, 0.004, 10.0, "r")]
LAYERS_3 = [(0.6, 0.0, 5.0, "b"), (0.8, -0.002, 8.0, "p"), (1.0, 0.004, 10.0, "r")]
CONFIG = (0, 1, 1, 4)  # TileBatch.config the autotuner settles on for the mixture


def listed():
    return [
        # a first look at a few fibers: launches and the call itself count
        {"name": "gen_small", "kind": "gen", "tissue": "crossing", "x": 48, "y": 40, "z": 24,
         "fibers": 40, "points": 8, "only_label": False},
        # one tile of the uneven mixture: every direction, odd sides
        {"name": "gen_tile", "kind": "gen", "tissue": "random", "x": 397, "y": 283, "z": 77,
         "fibers": 900, "points": 0, "only_label": False},
        # two crossing bundles at the size of a measured section
        {"name": "gen_crossing", "kind": "gen", "tissue": "crossing", "x": 512, "y": 512,
         "z": 120, "fibers": 2000, "points": 50, "only_label": False},
        # the voxelization-heavy volume: three layers, dense fibers
        {"name": "gen_watson", "kind": "gen", "tissue": "watson", "x": 1024, "y": 1024,
         "z": 240, "fibers": 20000, "points": 50, "only_label": False},
        # one image of a small volume
        {"name": "march_small", "kind": "march", "tissue": "crossing", "x": 48, "y": 40, "z": 24,
         "fibers": 40, "points": 8, "interpolate": "NN", "tilts": 1, "theta": 0.0, "phi": 0.0,
         "epa": False, "flip_z": False, "untilt": True, "step": 1.0},
        # one oblique image of an odd tile, interpolated the cheaper way, with
        # its transmittance, direction and retardation
        {"name": "march_tile_lerp", "kind": "march", "tissue": "random", "x": 397, "y": 283,
         "z": 77, "fibers": 900, "points": 0, "interpolate": "Lerp", "tilts": 1, "theta": 5.5,
         "phi": 90.0, "epa": True, "flip_z": False, "untilt": True, "step": 1.0},
        # the five images of a tilting series from one resident section
        {"name": "tilts_crossing", "kind": "march", "tissue": "crossing", "x": 512, "y": 512,
         "z": 120, "fibers": 2000, "points": 50, "interpolate": "Slerp", "tilts": 5,
         "theta": 5.5, "phi": 0.0, "epa": True, "flip_z": False, "untilt": True, "step": 1.0},
        # the untilted image of a large volume
        {"name": "march_flat_large", "kind": "march", "tissue": "crossing", "x": 1024, "y": 1024,
         "z": 240, "fibers": 4000, "points": 50, "interpolate": "Slerp", "tilts": 1,
         "theta": 0.0, "phi": 0.0, "epa": False, "flip_z": False, "untilt": True, "step": 1.0},
        # a batch of uneven tiles, voxelized and marched by one graph
        {"name": "batch_tiles", "kind": "batch", "tiles": 8, "first": 0, "tilts": 5,
         "interpolate": "Slerp", "epa": False},
        # a script's loop over the drop-in host API: tissue and five images as
        # numpy arrays
        {"name": "host_simpli", "kind": "host", "x": 256, "y": 256, "z": 60, "fibers": 500,
         "points": 26, "tilts": 5},
        # an image stack through the optics: blur and resample to the camera's
        # pixels, noise, epa of what the camera sees
        {"name": "optic_stack", "kind": "optic", "x": 512, "y": 512, "rho": 9, "sigma": 0.71,
         "scale": 0.2 / 1.33},
        # the tilt analysis of a tilting series at the camera's resolution
        {"name": "rofl_map", "kind": "rofl", "x": 160, "y": 150, "rho": 9, "grad": False,
         "masked": 0.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gen", "gen", "march", "march", "batch", "host", "optic", "rofl"])
    if kind in ("gen", "march"):
        tissue = rng.choice(["crossing", "random", "watson"])
        x, y, z = _log(rng, 40, 640), _log(rng, 40, 640), _log(rng, 20, 200)
        # about the fiber density of the listed volumes
        fibers = 2 * max(10, min(3000, int(x * y * z * rng.uniform(0.3, 1.2) / 16000)))
        case = {"kind": kind, "tissue": tissue, "x": x, "y": y, "z": z, "fibers": fibers,
                "points": 0 if tissue == "random" else rng.randint(6, 50)}
        if kind == "gen":
            return dict(case, only_label=rng.random() < 0.2)
        tilts = rng.choice([1, 1, 5])
        flat = tilts == 1 and rng.random() < 0.3
        return dict(case, interpolate=rng.choice(["NN", "Lerp", "Slerp", "Slerp"]), tilts=tilts,
                    theta=0.0 if flat else round(rng.uniform(1.0, 12.0), 2),
                    phi=0.0 if flat else round(rng.uniform(0.0, 360.0), 1),
                    epa=rng.random() < 0.5, flip_z=rng.random() < 0.25,
                    untilt=rng.random() < 0.8, step=rng.choice([1.0, 1.0, 1.0, 0.7]))
    if kind == "batch":
        return {"kind": "batch", "tiles": rng.randint(2, 8), "first": rng.randint(8, 248),
                "tilts": rng.choice([1, 5]), "interpolate": rng.choice(["Lerp", "Slerp", "Slerp"]),
                "epa": False}
    if kind == "host":
        x, y, z = _log(rng, 40, 256), _log(rng, 40, 256), _log(rng, 20, 60)
        return {"kind": "host", "x": x, "y": y, "z": z,
                "fibers": 2 * max(5, x * y * z // 16000), "points": rng.randint(8, 26),
                "tilts": rng.choice([1, 5])}
    if kind == "optic":
        return {"kind": "optic", "x": _log(rng, 40, 512), "y": _log(rng, 40, 512),
                "rho": rng.choice([6, 9]), "sigma": round(rng.uniform(0.4, 1.0), 2),
                "scale": rng.choice([0.2 / 1.33, 0.25, 0.5, round(rng.uniform(0.15, 1.0), 3)])}
    return {"kind": "rofl", "x": _log(rng, 16, 110), "y": _log(rng, 16, 110),
            "rho": rng.choice([6, 9]), "grad": rng.random() < 0.3,
            "masked": rng.choice([0.0, 0.0, 0.4])}


# ------------------------------------------------------------------ inputs ---
def _random_fibers(rng, dim, n, voxel_size, segment_um=2.0):
    """``n`` straight fibers in uniformly random directions through uniformly
    random points of the volume, cut into segments of about 2 um."""
    size = np.asarray(dim) * voxel_size
    v = rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    c = rng.uniform(0, 1, (n, 3)) * size
    r = rng.lognormal(np.log(1.0), 0.2, n)
    a, b = (0.0 - c) / v, (size - c) / v
    t0 = np.minimum(a, b).max(1) - r
    t1 = np.maximum(a, b).min(1) + r
    fibers = []
    for k in range(n):
        t = np.linspace(t0[k], t1[k], max(2, int(np.ceil((t1[k] - t0[k]) / segment_um)) + 1))
        fibers.append(np.c_[c[k] + t[:, None] * v[k], np.full(t.size, r[k])])
    return fibers


def _tissue(case, seed):
    """The case's volume with its fibers and layers (synth.Workload)."""
    dim = (case["x"], case["y"], case["z"])
    n = case["fibers"]
    if case["tissue"] == "crossing":
        return synth.crossing(seed=seed, n_per_bundle=n // 2, dim=dim, n_points=case["points"])
    if case["tissue"] == "watson":
        return synth.watson(seed=seed, n_fibers=n, dim=dim, n_points=case["points"])
    rng = np.random.default_rng(seed)
    return synth.Workload("random", dim, 0.2, [_random_fibers(rng, dim, n, 0.2)], [LAYERS_2])


def _tiles(case, seed):
    """Tiles of the uneven mixture: its sizes, fiber counts, dn and mu."""
    rng = np.random.default_rng(seed)
    tiles = []
    for i in range(case["tiles"]):
        dim, n, dn, mu = synth.tile_params(case["first"] + i)
        layers = [(0.75, 0.0, mu, "b"), (1.0, dn, mu, "r")]
        tiles.append(synth.Workload("tile", dim, 0.2, [_random_fibers(rng, dim, n, 0.2)],
                                    [layers], tilts=synth.TILTS_5[: case["tilts"]]))
    return tiles


def _generator(w):
    g = _Generator()
    g.set_volume(w.dim, w.origin, w.voxel_size)
    g.set_fiber_bundles(w.bundles, w.layers)
    return g


def _setup(case, w):
    """Keyword arguments of _Simulator.set_pli_setup."""
    return dict(synth.OPTICS, voxel_size=w.voxel_size, interpolate=case["interpolate"],
                filter_rotations=synth.ROT_9, flip_z=case.get("flip_z", False),
                untilt_sensor_view=case.get("untilt", True), step_size=case.get("step", 1.0))


def _tilts(case):
    if case["tilts"] == 1:
        return np.deg2rad([(case["theta"], case["phi"])])
    phis = case["phi"] + np.arange(4) * 90.0
    return np.deg2rad([(0.0, 0.0)] + [(case["theta"], p) for p in phis])


def _series(case, seed):
    """A tilting series [5, X, Y, rho] as the camera gives it: uniform
    orientations and retardations, the gain's noise."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n = (case["x"], case["y"])

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)

    phi, alpha = uniform(0, math.pi), uniform(-1.2, 1.2)
    t_rel, trans = uniform(0.05, 0.8), uniform(3000.0, 9000.0)
    rho = torch.arange(case["rho"], device="cuda", dtype=torch.float64) * (math.pi / case["rho"])
    axis = torch.stack([alpha.cos() * phi.cos(), alpha.cos() * phi.sin(), alpha.sin()])
    out = []
    for theta, psi in synth.TILTS_5:
        rot = torch.tensor(_rot_zyz(psi, theta, -psi), device="cuda")
        v = torch.einsum("ij,jxy->ixy", rot, axis)
        q = v[0] ** 2 + v[1] ** 2
        ret = torch.sin(0.5 * math.pi * t_rel / math.cos(theta) * q)
        p = torch.atan2(v[1], v[0])
        image = trans[..., None] * (1 + ret[..., None] * torch.sin(2 * (rho - p[..., None])))
        noise = torch.randn(image.shape, generator=gen, device="cuda", dtype=torch.float64)
        out.append((image + (3.0 * image.clamp_min(1.0)).sqrt() * noise).clamp_min(1.0))
    return torch.stack(out)


def _stack(case, seed):
    """A march's image stack [X, Y, rho]: smooth structure and fine texture."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (case["x"], case["y"], case["rho"])
    fine = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
    x = torch.arange(case["x"], device="cuda", dtype=torch.float64)[:, None, None]
    y = torch.arange(case["y"], device="cuda", dtype=torch.float64)[None, :, None]
    rho = torch.arange(case["rho"], device="cuda", dtype=torch.float64) * (math.pi / case["rho"])
    return 4000 + 1500 * torch.sin(2 * (rho - x / 37 - y / 53)) + 1000 * fine


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gen":
        w = _tissue(case, seed)
        return {"case": case, "workload": w, "gen": _generator(w)}
    if kind == "march":
        w = _tissue(case, seed)
        label, vector, props, _ = _generator(w).run_generation_device()
        props = props.copy()
        s = _setup(case, w)
        sim = _Simulator()
        sim.set_pli_setup(s["step_size"], s["light_intensity"], s["voxel_size"], s["wavelength"],
                          s["tissue_refrection"], s["interpolate"], s["untilt_sensor_view"],
                          s["flip_z"], s["filter_rotations"])
        return {"case": case, "sim": sim, "setup": s, "dim": w.dim, "label": label,
                "vector": vector, "props": props, "tilts": _tilts(case)}
    if kind == "batch":
        tiles = _tiles(case, seed)
        batch = TileBatch(tiles, _setup(case, tiles[0]), epa=case["epa"])
        batch.config = CONFIG
        batch.set_shape(CONFIG[3])
        batch.allocate()
        batch.capture()
        return {"case": case, "tiles": tiles, "batch": batch}
    if kind == "host":
        w = _tissue(dict(case, tissue="crossing"), seed)
        s = Simpli()
        s.voxel_size = w.voxel_size
        s.dim = w.dim
        s.dim_origin = w.origin
        s.fiber_bundles = w.bundles
        s.fiber_bundles.layers = w.layers
        s.filter_rotations = synth.ROT_9
        s.interpolate = "Slerp"
        s.wavelength = synth.OPTICS["wavelength"]
        s.light_intensity = synth.OPTICS["light_intensity"]
        s.tilts = synth.TILTS_5[: case["tilts"]]
        return {"case": case, "workload": w, "simpli": s}
    if kind == "optic":
        return {"case": case, "image": _stack(case, seed), "seed": int(seed)}
    data = _series(case, seed)
    mask = None
    if case["masked"]:
        gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        mask = torch.rand(data.shape[1:3], generator=gen, device="cuda") >= case["masked"]
    return {"case": case, "data": data, "mask": mask}


# -------------------------------------------------------------------- pass ---
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gen":
        label, vector, props, _ = state["gen"].run_generation_device(
            only_label=case["only_label"])
        return {"label": label, "vector": vector, "props": props}
    if kind == "march":
        sim, tilts = state["sim"], state["tilts"]
        args = (state["dim"], state["label"], state["vector"], state["props"])
        if len(tilts) == 1:
            out = [sim.run_simulation_device(*args, float(tilts[0, 0]), float(tilts[0, 1]),
                                             epa=case["epa"])]
        else:
            out = sim.run_tilts_device(*args, tilts, epa=case["epa"])
        return [list(o) if case["epa"] else [o] for o in out]
    if kind == "batch":
        b = state["batch"]
        b.replay()
        return {"labels": [b.label(t) for t in range(len(state["tiles"]))],
                "vectors": [b.vector(t) for t in range(len(state["tiles"]))],
                "images": [b.image(p) for p in range(int(b.info.n_pairs))]}
    if kind == "host":
        s = state["simpli"]
        tissue, axis, props = s.generate_tissue()
        images = [s.run_simulation(tissue, axis, props, theta, phi) for theta, phi in s.tilts]
        return {"tissue": tissue, "axis": axis, "props": props, "images": images}
    if kind == "optic":
        res = optic.filter_resample_device(state["image"], case["sigma"], case["scale"])
        # a seed per pass, as a pipeline that has to be repeatable gives it
        noisy = optic.NegativeBinomialNoise(3.0, seed=state["seed"]).device(res)
        return {"resampled": res, "noisy": noisy, "epa": list(optic.epa_device(noisy))}
    return analysis.rofl_device(state["data"], grad_mode=case["grad"], mask=state["mask"])


def work(case):
    kind = case["kind"]
    if kind == "gen":
        n = case["x"] * case["y"] * case["z"]
        return {"bytes": n * (4 if case["only_label"] else 16) + 32 * case["fibers"] * 30,
                "flops": 25 * n}
    if kind in ("march", "host"):
        pixels = case["x"] * case["y"]
        n, tilts = pixels * case["z"], case["tilts"]
        images = 72 * pixels * tilts
        if kind == "host":  # tissue out, tissue in again for each image, images out
            return {"bytes": 16 * n * (1 + tilts) + images, "flops": (25 + 40 * tilts) * n}
        return {"bytes": 16 * n + images + (24 * pixels * tilts if case["epa"] else 0),
                "flops": 40 * n * tilts}
    if kind == "batch":
        n = pixels = 0
        for i in range(case["tiles"]):
            x, y, z = synth.tile_params(case["first"] + i)[0]
            n, pixels = n + x * y * z, pixels + x * y
        return {"bytes": 2 * 16 * n + 72 * pixels * case["tilts"],
                "flops": (25 + 40 * case["tilts"]) * n}
    n = case["x"] * case["y"] * case["rho"]
    if kind == "optic":
        out = n * case["scale"] ** 2
        taps = 2 * int(4 * case["sigma"] / case["scale"] + 0.5) + 1 / case["scale"]
        return {"bytes": 8 * n + 3 * 8 * out,
                "flops": 2 * taps * n * case["scale"] * (1 + case["scale"])}
    pixels = case["x"] * case["y"] * (1 - case["masked"])
    # about 25 evaluations of the model after a 6 x 6 start grid
    return {"bytes": 5 * 8 * n + 64 * case["x"] * case["y"],
            "flops": pixels * 5 * case["rho"] * (6 + 25) * 30}


# ------------------------------------------------------------ 64-bit values ---
def _rot_zyz(g, b, a):
    def rz(t):
        return np.array([[math.cos(t), -math.sin(t), 0], [math.sin(t), math.cos(t), 0],
                         [0, 0, 1.0]])

    ry = np.array([[math.cos(b), 0, math.sin(b)], [0, 1.0, 0], [-math.sin(b), 0, math.cos(b)]])
    return rz(g) @ ry @ rz(a)


def _segments(w):
    """Segment starts, ends and radii in voxels, and their bundle."""
    p, q, r0, r1, bundle = [], [], [], [], []
    f = 1.0 / w.voxel_size
    for b, fibers in enumerate(w.bundles):
        for fiber in fibers:
            x = (fiber[:, :3] - w.origin) * f if np.any(w.origin) else fiber[:, :3] * f
            r = fiber[:, 3] * f
            p.append(x[:-1])
            q.append(x[1:])
            r0.append(r[:-1])
            r1.append(r[1:])
            bundle.append(np.full(len(x) - 1, b))
    cat = [torch.from_numpy(np.concatenate(a)).cuda() for a in (p, q, r0, r1, bundle)]
    return cat


def _closest(pt, p, q, r0, r1):
    """Offset from each point to the closest point of its segment, and the
    fiber's radius there."""
    v, w = q - p, pt - p
    c1, c2 = (w * v).sum(1), (v * v).sum(1)
    t = torch.where(c1 < 0, torch.zeros_like(c1), torch.where(c2 <= c1, torch.ones_like(c1),
                                                              c1 / c2))
    return p + v * t[:, None] - pt, r0 * (1 - t) + r1 * t


def _voxelize64(w):
    """The orientation field of the volume in 64 bits, flat [n, 3]."""
    X, Y, Z = (int(d) for d in w.dim)
    p, q, r0, r1, bundle = _segments(w)
    dev = p.device
    outer = torch.tensor([max(ly[0] for ly in lys) ** 2 for lys in w.layers], device=dev,
                         dtype=torch.float64)
    rmax = (torch.maximum(r0, r1) * outer.sqrt()[bundle])[:, None]
    top = torch.tensor([X, Y, Z], device=dev, dtype=torch.float64)
    lo = torch.minimum(p, q).sub(rmax).clamp_min(0).minimum(top).to(torch.int64)
    hi = torch.maximum(p, q).add(rmax).minimum(top).clamp_min(0).add(0.5).to(torch.int64)
    ext = (hi.minimum(top.to(torch.int64)) - lo).clamp_min(0)
    count = ext.prod(1)
    # fibers whose box misses the volume have an empty box here too
    key = torch.full((X * Y * Z,), 2 ** 63 - 1, device=dev, dtype=torch.int64)
    ends = torch.cumsum(count, 0).cpu().numpy()
    a = 0
    while a < len(ends):
        done = ends[a - 1] if a else 0
        b = max(a + 1, int(np.searchsorted(ends, done + 12_000_000)))
        seg = torch.repeat_interleave(torch.arange(a, b, device=dev), count[a:b])
        first = torch.cumsum(count[a:b], 0) - count[a:b]
        k = torch.arange(seg.numel(), device=dev) - first[seg - a]
        e = ext[seg]
        z, k = k % e[:, 2], k // e[:, 2]
        y, x = k % e[:, 1], k // e[:, 1]
        ijk = torch.stack([x, y, z], 1) + lo[seg]
        d, r = _closest(ijk.double() + 0.5, p[seg], q[seg], r0[seg], r1[seg])
        dist = (d * d).sum(1).float()
        ok = dist <= outer.float()[bundle[seg]] * (r * r).float()
        flat = (ijk[:, 0] * Y + ijk[:, 1]) * Z + ijk[:, 2]
        keys = (dist.view(torch.int32).to(torch.int64) << 32) | (0xFFFFFFFF - seg)
        key.scatter_reduce_(0, flat[ok], keys[ok], "amin")
        a = b
    out = torch.zeros((X * Y * Z, 3), device=dev, dtype=torch.float64)
    at = (key < 2 ** 63 - 1).nonzero()[:, 0]
    for at in torch.split(at, 12_000_000):
        seg = 0xFFFFFFFF - (key[at] & 0xFFFFFFFF)
        ijk = torch.stack([at // (Y * Z), at // Z % Y, at % Z], 1).double() + 0.5
        d, r = _closest(ijk, p[seg], q[seg], r0[seg], r1[seg])
        dist = (key[at] >> 32).to(torch.int32).view(torch.float32)
        quot = (dist / (r * r).float()).double()
        radial = -d / d.norm(dim=1, keepdim=True).clamp_min(1e-300)
        along = q[seg] - p[seg]
        along = along / along.norm(dim=1, keepdim=True).clamp_min(1e-300)
        v = torch.zeros_like(d)
        for b, lys in enumerate(w.layers):
            lys = sorted(lys)
            below = -1.0
            for scale, _, _, model in lys:
                inside = (bundle[seg] == b) & (quot > below) & (quot <= scale * scale)
                below = scale * scale
                if model != "b":
                    v = torch.where(inside[:, None], radial if model == "r" else along, v)
        out[at] = v
    return out


def _props64(w):
    most = max(len(lys) for lys in w.layers)
    props = np.zeros((1 + most * len(w.layers), 2))
    for b, lys in enumerate(w.layers):
        for i, (_, dn, mu, model) in enumerate(sorted(lys)):
            props[1 + i + b * most] = (0.0 if model == "b" else dn, mu)
    return props


def _lerp64(v, u, t):
    a, b = v * (1 - t), u * t
    out = torch.where(((a * b).sum(-1) >= 0)[..., None], a + b, a - b)
    return _with_zeros(v, u, out)


def _slerp64(v, u, t):
    flipped = torch.where(((v * u).sum(-1) < 0)[..., None], -u, u)
    c = (v * flipped).sum(-1) / (v.norm(dim=-1) * flipped.norm(dim=-1))
    th = torch.arccos(c.clamp(-1, 1))[..., None]
    out = (v * torch.sin((1 - t) * th) + flipped * torch.sin(t * th)) / torch.sin(th)
    same = ((v - flipped) ** 2).sum(-1) < 1e-12
    return _with_zeros(v, u, torch.where(same[..., None], v, out))


def _with_zeros(v, u, out):
    out = torch.where((u == 0).all(-1)[..., None], v, out)
    return torch.where((v == 0).all(-1)[..., None], u, out)


def _march64(label, vector, props, setup, theta, phi):
    """The image stack [X, Y, rho] in 64 bits: every ray steps through the
    volume with the state of its polarisation in the frame of the filter."""
    X, Y, Z = (int(d) for d in label.shape)
    dev = label.device
    label, vector = label.reshape(-1), vector.reshape(-1, 3)
    step = setup["step_size"]
    thick = setup["voxel_size"] * 1e-6 * step
    props = torch.tensor(np.asarray(props), device=dev, dtype=torch.float64)
    dn, mu = props[:, 0], props[:, 1]
    retard = (math.pi / 2) * (dn * 4 * thick / (setup["wavelength"] * 1e-9))
    absorb = mu * 1e3 * thick
    way = np.array([math.cos(phi) * math.sin(theta), math.sin(phi) * math.sin(theta),
                    math.cos(theta)])
    way[np.abs(way) < 1e-15] = 0.0
    rot = torch.tensor(_rot_zyz(phi, theta, -phi), device=dev)
    shift = way / math.cos(theta) * Z
    cx = torch.arange(X, device=dev, dtype=torch.float64).add(0.5)[:, None].expand(X, Y)
    cy = torch.arange(Y, device=dev, dtype=torch.float64).add(0.5)[None, :].expand(X, Y)
    if setup["untilt_sensor_view"]:
        x, y = cx - 0.5 * shift[0], cy - 0.5 * shift[1]
    else:  # the camera's pixels seen through the tilted section
        ang = math.asin(math.sin(-theta) * setup["tissue_refrection"])
        pc = np.array([X, Y, Z]) * 0.5
        m, back = _rot_zyz(phi, ang, -phi), _rot_zyz(phi, -ang, -phi)
        pt = m @ np.array([-pc[0], -pc[1], pc[2]])
        e, f = cx - pc[0] - pt[0], cy - pc[1] - pt[1]
        det = m[0, 0] * m[1, 1] - m[1, 0] * m[0, 1]
        s = (e * m[1, 1] - f * m[0, 1]) / det
        t = (m[0, 0] * f - m[1, 0] * e) / det
        rel = [pt[i] + m[i, 0] * s + m[i, 1] * t for i in range(3)]
        x, y = (sum(back[i, j] * rel[j] for j in range(3)) + pc[i] - shift[i] for i in range(2))
    x = (x + 0.5 * step * way[0]).reshape(-1)
    y = (y + 0.5 * step * way[1]).reshape(-1)
    z = 0.5 * step * way[2]
    mix = {"Lerp": _lerp64, "Slerp": _slerp64}.get(setup["interpolate"])
    u1 = torch.zeros(X * Y, device=dev, dtype=torch.float64)
    u2, u3, gone = u1.clone(), u1 - 1, u1.clone()

    def mirrored(iz):
        return Z - 1 - iz if setup["flip_z"] else iz

    while math.floor(z) < Z:
        ix, iy = x.floor().long(), y.floor().long()
        ray = ((ix >= 0) & (ix < X) & (iy >= 0) & (iy < Y)).nonzero()[:, 0]
        lab = label[(ix[ray] * Y + iy[ray]) * Z + mirrored(math.floor(z))].long()
        bent = (dn[lab] != 0) & (lab != 0)
        plain = ray[~bent]
        gone[plain] = gone[plain] + absorb[lab[~bent]]
        ray, lab = ray[bent], lab[bent]
        if mix is None:
            v = vector[(ix[ray] * Y + iy[ray]) * Z + mirrored(math.floor(z))].double()
        else:
            hx, hy, hz = x[ray] - 0.5, y[ray] - 0.5, z - 0.5
            x0, y0, z0 = hx.floor(), hy.floor(), math.floor(hz)
            xs = [c.long().clamp(0, X - 1) for c in (x0, hx.ceil())]
            ys = [c.long().clamp(0, Y - 1) for c in (y0, hy.ceil())]
            zs = [mirrored(min(max(c, 0), Z - 1)) for c in (z0, math.ceil(hz))]
            corner = []
            for k in range(8):
                at = (xs[k & 1] * Y + ys[k >> 1 & 1]) * Z + zs[k >> 2]
                corner.append(vector[at].double() * (label[at].long() == lab)[:, None])
            td = (hx - x0)[:, None]
            c00, c10, c01, c11 = (mix(corner[k], corner[k + 1], td) for k in (0, 2, 4, 6))
            td = (hy - y0)[:, None]
            v = mix(mix(c00, c10, td), mix(c01, c11, td), hz - z0)
        n2 = (v * v).sum(1)
        some = n2 > 0
        ray, lab, v, n2 = ray[some], lab[some], v[some], n2[some]
        v = v @ rot.T
        q = v[:, 0] ** 2 + v[:, 1] ** 2
        ret = retard[lab] * q / n2.sqrt()
        safe = torch.where(q > 0, q, torch.ones_like(q))
        c = torch.where(q > 0, (v[:, 0] ** 2 - v[:, 1] ** 2) / safe, torch.ones_like(q))
        s = 2 * v[:, 0] * v[:, 1] / safe
        a, b, w = u1[ray], u2[ray], u3[ray]
        a1, c1 = a * c - b * s, a * s + b * c
        b1 = c1 * ret.cos() + w * ret.sin()
        u3[ray] = w * ret.cos() - c1 * ret.sin()
        u1[ray] = a1 * c + b1 * s
        u2[ray] = b1 * c - a1 * s
        gone[ray] = gone[ray] + absorb[lab]
        x, y, z = x + step * way[0], y + step * way[1], z + step * way[2]
    rho = torch.tensor(np.asarray(setup["filter_rotations"]), device=dev)
    image = (setup["light_intensity"] / 4 * torch.exp(-gone))[:, None] * (
        1 - u1[:, None] * torch.cos(2 * rho) + u2[:, None] * torch.sin(2 * rho))
    return image.reshape(X, Y, -1)


def _epa64(image):
    n = image.shape[-1]
    rho2 = 2 * torch.arange(n, device=image.device, dtype=torch.float64) * (math.pi / n)
    a0 = image.mean(-1)
    a1, b1 = 2 * (image * rho2.sin()).mean(-1), 2 * (image * rho2.cos()).mean(-1)
    return [2 * a0, torch.remainder(0.5 * torch.atan2(-b1, a1) + math.pi, math.pi),
            (a1 * a1 + b1 * b1).sqrt() / torch.where(a0 < 2.2e-14, torch.ones_like(a0), a0)]


def _blur64(image, sd, axis):
    n = image.shape[axis]
    radius = int(4 * sd + 0.5)
    k = np.arange(-radius, radius + 1)
    weight = np.exp(-0.5 / (sd * sd) * k.astype(float) ** 2)
    weight /= weight.sum()
    out = torch.zeros_like(image)
    for j, wj in zip(k, weight):
        at = np.mod(np.arange(n) + j, 2 * n)
        at = torch.from_numpy(np.where(at < n, at, 2 * n - 1 - at)).to(image.device)
        out = out + wj * image.index_select(axis, at)
    return out


def _resample64(image, scale, axis):
    n = image.shape[axis]
    size = int(round(n * scale))
    at = np.floor((np.arange(n) + 0.5) * scale).astype(np.int64)
    keep = at < size
    at, src = torch.from_numpy(at[keep]).to(image.device), torch.from_numpy(np.nonzero(keep)[0])
    shape = list(image.shape)
    shape[axis] = size
    total = torch.zeros(shape, device=image.device, dtype=torch.float64)
    total.index_add_(axis, at, image.index_select(axis, src.to(image.device)))
    count = torch.bincount(at, minlength=size).double()
    return total / count.reshape([-1 if i == axis else 1 for i in range(3)])


def exact(case, seed):
    kind = case["kind"]
    if kind == "gen":
        w = _tissue(case, seed)
        vector = None if case["only_label"] else _voxelize64(w).reshape(*w.dim.tolist(), 3)
        return {"label": None, "vector": vector, "props": _props64(w)}
    if kind == "march":
        s = prepare(case, seed)  # the tissue that the images are of
        out = []
        for theta, phi in s["tilts"]:
            image = _march64(s["label"], s["vector"], s["props"], s["setup"], theta, phi)
            # the direction is an angle mod pi: no value where it may wrap
            epa = _epa64(image) if case["epa"] else []
            out.append([image] + (epa[:1] + [None] + epa[2:] if epa else []))
        return out
    if kind == "batch":
        s = prepare(case, seed)
        s["batch"].replay()
        vectors, images = [], []
        for t, w in enumerate(s["tiles"]):
            vectors.append(_voxelize64(w).reshape(*w.dim.tolist(), 3))
            label, vector = s["batch"].label(t), s["batch"].vector(t)
            images += [_march64(label, vector, _props64(w), _setup(case, w), theta, phi)
                       for theta, phi in w.tilts]
        return {"labels": [None] * len(vectors), "vectors": vectors, "images": images}
    if kind == "host":
        w = _tissue(dict(case, tissue="crossing"), seed)
        label, _, props, _ = _generator(w).run_generation_device()
        axis = _voxelize64(w).reshape(*w.dim.tolist(), 3)
        setup = _setup(dict(case, interpolate="Slerp"), w)
        images = [_march64(label, axis.float(), props, setup, theta, phi).cpu().numpy()
                  for theta, phi in synth.TILTS_5[: case["tilts"]]]
        return {"tissue": None, "axis": axis.cpu().numpy(), "props": _props64(w),
                "images": images}
    if kind == "optic":
        image, sd = _stack(case, seed), case["sigma"] / case["scale"]
        image = _blur64(_blur64(image, sd, 0), sd, 1)
        res = _resample64(_resample64(image, case["scale"], 0), case["scale"], 1)
        return {"resampled": res, "noisy": None, "epa": None}
    return None  # a fit by forward differences: its last steps are rounding
