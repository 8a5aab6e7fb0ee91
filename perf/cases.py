"""Benchmark cases of the Tb.Th / Tb.Sp path: what users of this package call.

Each case goes through the package's public entry points: ``analyze_thickness``
(device and host inputs, the feature modes, with and without maps),
``local_thickness`` and ``euclidean_distance_transform_squared`` in both
phases, ``nonzero_stats``, ``volume_metrics`` and the batched form.  Volumes
come from the package's own synthetic generator: Gaussian-smoothed noise
thresholded at a bone fraction, with a cylinder or sphere ROI.
"""

import math

import numpy as np
import torch

import bone_morphometry_gb300 as bm
from bone_morphometry_gb300 import serving
from bone_morphometry_gb300 import synthetic


def _tbth(name, shape, sigma, bvtv, roi, radius, spacing, mode="classic", maps=False, host=False):
    d, h, w = shape
    sx, sy, sz = sigma if isinstance(sigma, tuple) else (sigma, sigma, sigma)
    return dict(name=name, kind="tbth", d=d, h=h, w=w, sx=sx, sy=sy, sz=sz, bvtv=bvtv, roi=roi, radius=radius,
                spacing=spacing, mode=mode, maps=maps, host=host)


def _field(name, kind, shape, sigma, bvtv, phase="foreground", squared=False):
    d, h, w = shape
    return dict(name=name, kind=kind, d=d, h=h, w=w, sx=sigma, sy=sigma, sz=sigma, bvtv=bvtv, phase=phase,
                squared=squared)


def listed():
    return [
        # A cropped sub-volume, one of many in a region-of-interest study: launches and latency count.
        _tbth("tbth_64", (72, 56, 64), 2.5, 0.25, "cylinder", 25.0, 10.0),
        # The small scan of the package's own configurations, called as a script does: numpy arrays
        # as they come from the image reader, with the quantiles.
        _tbth("tbth_128_host_quantiles", (128, 128, 128), 3.0, 0.25, "cylinder", 56.0, 10.0, mode="standard",
              host=True),
        # One ordinary specimen on the device: the package's headline workload.
        _tbth("tbth_512", (512, 512, 512), 5.0, 0.15, "cylinder", 240.0, 19.5),
        # One large plate-like specimen: the package's largest single-volume workload.
        _tbth("tbth_1024", (1024, 1024, 1024), (4.0, 4.0, 8.0), 0.30, "sphere", 500.0, 8.0),
        # A specimen of odd sizes whose thickness maps are kept for display, with quantiles.
        _tbth("tbth_ragged_maps", (251, 187, 203), 4.0, 0.30, "cylinder", 84.0, 12.5, mode="experimental", maps=True),
        # Local thickness of a segmented trabecula crop, odd sizes.
        _field("thickness_fg_small", "lt", (70, 81, 97), 2.5, 0.30),
        # Local thickness of the pore space of a whole crop (no ROI), with the squared radii, odd sizes.
        _field("thickness_bg_ragged", "lt", (301, 190, 253), 4.0, 0.25, phase="background", squared=True),
        # The distance field of the background that the surface and orientation measures read, odd sizes.
        _field("edt_bg_ragged", "edt", (417, 333, 379), 5.0, 0.20, phase="background"),
        # The distance field of the bone phase of an ordinary specimen.
        _field("edt_fg_512", "edt", (512, 512, 512), 5.0, 0.15),
        # Statistics with quantiles of a thickness map that a program already holds.
        dict(name="stats_320", kind="stats", d=320, h=311, w=337, fill=0.35, scale=12.0, quantiles=True),
        # Bone volume fraction and ROI-boundary bone fraction of an ordinary specimen, odd sizes.
        dict(name="volume_ragged", kind="volume", d=430, h=389, w=401, sx=4.0, sy=4.0, sz=4.0, bvtv=0.2, spacing=10.0),
        # A study's specimens of uneven sizes, from host arrays through the batched form.
        dict(name="batch_16", kind="batch", n=16, lo=96, hi=384, mix=1004),
    ]


def _edges(rng, lo, hi):
    return tuple(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["tbth", "tbth", "tbth", "lt", "lt", "edt", "edt", "stats", "volume", "batch"])
    if kind == "batch":
        return dict(kind="batch", n=rng.randint(3, 16), lo=64, hi=384, mix=rng.randint(1, 10**6))
    shape = _edges(rng, 48, 640)
    if kind == "stats":
        d, h, w = shape
        return dict(kind="stats", d=d, h=h, w=w, fill=rng.uniform(0.05, 0.9), scale=rng.uniform(5.0, 25.0),
                    quantiles=rng.random() < 0.7)
    # structures from 2 voxels up, and several of them across the shortest edge
    sigma = rng.uniform(2.0, min(8.0, max(2.5, min(shape) / 20.0)))
    bvtv = rng.uniform(0.15, 0.40) if min(shape) < 96 else rng.uniform(0.08, 0.40)
    d, h, w = shape
    if kind == "volume":
        return dict(kind="volume", d=d, h=h, w=w, sx=sigma, sy=sigma, sz=sigma, bvtv=bvtv,
                    spacing=rng.uniform(5.0, 25.0))
    if kind == "tbth":
        c = _tbth("", shape, sigma, bvtv, rng.choice(["cylinder", "cylinder", "sphere"]), 0.47 * min(shape),
                  rng.uniform(5.0, 25.0), mode=rng.choice(["classic", "standard", "bonej", "experimental"]),
                  maps=rng.random() < 0.25, host=rng.random() < 0.4)
    else:
        c = _field("", kind, shape, sigma, bvtv, phase=rng.choice(["foreground", "background"]),
                   squared=rng.random() < 0.4)
    del c["name"]
    return c


def _specimen(case, seed, roi="all", radius=0.0, spacing=1.0):
    return synthetic.make_specimen_torch((case["d"], case["h"], case["w"]), (case["sx"], case["sy"], case["sz"]),
                                         case["bvtv"], roi, radius, spacing, seed, to_host=False)


def _batch_specs(case, seed):
    specs = synthetic.batch_specs(case["n"], case["lo"], case["hi"], seed=case["mix"])
    return [(s, (seed * 1009 + i) & 0x7FFFFFFF) for i, s in enumerate(specs)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        items = []
        for s, item_seed in _batch_specs(case, seed):
            d, h, w = s.shape
            sp = synthetic.make_specimen_torch(s.shape, s.sigma, max(s.bvtv, 0.15), "cylinder", 0.45 * min(w, h),
                                               s.spacing_um, item_seed)
            items.append(serving.SpecimenInput(sp.bone, sp.roi, s.spacing_um))
        return dict(case=case, items=items)
    if kind == "stats":
        # diameters of a thickness map: 2 * sqrt of whole squared radii, smoothed entries between them, zero off-phase
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        n = case["d"] * case["h"] * case["w"]
        r2 = torch.randint(1, 900, (n,), generator=g, device="cuda")
        v = 2.0 * torch.sqrt(r2.to(torch.float32))
        mix = torch.rand((n,), generator=g, device="cuda")
        v = torch.where(mix < 0.3, v * (0.8 + mix), v)
        v = torch.where(torch.rand((n,), generator=g, device="cuda") < case["fill"], v, torch.zeros_like(v))
        return dict(case=case, values=v.view(case["d"], case["h"], case["w"]).contiguous())
    if kind == "tbth":
        sp = _specimen(case, seed, case["roi"], case["radius"], case["spacing"])
        bone, roi = sp.bone, sp.roi
        if case["host"]:
            bone, roi = bone.cpu().numpy(), roi.cpu().numpy()
        return dict(case=case, bone=bone, roi=roi, mode=bm.FeatureMode(case["mode"]))
    if kind == "volume":
        sp = _specimen(case, seed, "cylinder", 0.45 * min(case["h"], case["w"]), case["spacing"])
        return dict(case=case, bone=sp.bone, roi=sp.roi)
    sp = _specimen(case, seed)
    phase = bm.Phase.BACKGROUND if case["phase"] == "background" else bm.Phase.FOREGROUND
    return dict(case=case, volume=sp.bone, phase=phase)


_STATS = ("count", "mean", "standard_deviation", "maximum", "coefficient_of_variation", "sum", "sum_of_squares")
_QUANTILES = ("median", "percentile_10", "percentile_25", "percentile_75", "percentile_90", "interquartile_range")


def _stats_dict(s, quantiles):
    return {k: getattr(s, k) for k in _STATS + (_QUANTILES if quantiles else ())}


def _wants_quantiles(mode):
    return mode in ("standard", "experimental")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tbth":
        r = bm.analyze_thickness(state["bone"], state["roi"], case["spacing"], state["mode"],
                                 return_maps=case["maps"])
        q = _wants_quantiles(case["mode"])
        out = dict(thickness=_stats_dict(r.thickness, q), spacing=_stats_dict(r.spacing, q))
        if case["maps"]:
            out["thickness_map"], out["spacing_map"] = r.thickness_map, r.spacing_map
        return out
    if kind == "lt":
        r = bm.local_thickness(state["volume"], state["phase"], return_squared=case["squared"])
        return dict(map=r[0], squared=r[1]) if case["squared"] else dict(map=r)
    if kind == "edt":
        return bm.euclidean_distance_transform_squared(state["volume"], state["phase"])
    if kind == "stats":
        return _stats_dict(bm.nonzero_stats(state["values"], case["scale"], case["quantiles"]), case["quantiles"])
    if kind == "volume":
        m = bm.volume_metrics(state["bone"], state["roi"], case["spacing"])
        return [m.bone_voxels, m.roi_voxels, m.boundary_bone_voxels, m.bone_volume, m.total_volume,
                m.bone_volume_fraction, m.roi_boundary_bone_fraction]
    res = serving.batch_tbth_tbsp(state["items"])
    rows = lambda s: [getattr(s, k) for k in _STATS if k != "count"]
    return dict(thickness=np.array([rows(th) for th, _, _ in res]), spacing=np.array([rows(sp) for _, sp, _ in res]),
                counts=np.array([(th.count, sp.count) for th, sp, _ in res]),
                status=np.array([st for _, _, st in res]))


def work(case):
    """Input bytes read once and output bytes written once; the path is integer work, so no flops are counted."""
    kind = case["kind"]
    if kind == "batch":
        specs = synthetic.batch_specs(case["n"], case["lo"], case["hi"], seed=case["mix"])
        return {"bytes": 2 * sum(int(np.prod(s.shape)) for s in specs), "flops": 0}
    n = case["d"] * case["h"] * case["w"]
    if kind == "tbth":
        return {"bytes": 2 * n + (8 * n if case["maps"] else 0), "flops": 0}
    if kind == "lt":
        return {"bytes": n + 4 * n + (4 * n if case["squared"] else 0), "flops": 0}
    return {"bytes": {"edt": 5 * n, "stats": 4 * n, "volume": 2 * n}[kind], "flops": 0}


# ---- the same results from plain torch in 64 bits ------------------------------------------

_EXACT_VOXELS = 4 << 20  # larger volumes take too long this way


def _shifted(a, axis, s, fill):
    """a moved by s along axis, the vacated entries filled."""
    out = torch.full_like(a, fill)
    n = a.shape[axis]
    if abs(s) < n:
        src = a.narrow(axis, max(0, -s), n - abs(s))
        out.narrow(axis, max(0, s), n - abs(s)).copy_(src)
    return out


def _dist_sq(sites, limit=None):
    """Squared distance to the nearest site (up to `limit` voxels along each axis)."""
    far = 1 << 40
    g = torch.where(sites, 0, far)
    for axis in range(3):
        best = g.clone()
        for s in range(1, min(g.shape[axis] - 1, limit if limit is not None else 1 << 30) + 1):
            best = torch.minimum(best, _shifted(g, axis, s, far) + s * s)
            best = torch.minimum(best, _shifted(g, axis, -s, far) + s * s)
        g = best
    return g


def _thickness_exact(mask):
    """(map, squared): local thickness in f64 and the squared radius of the largest covering ball."""
    r2 = torch.where(mask, _dist_sq(~mask), 0)
    ball = torch.zeros_like(r2)
    for v in torch.unique(r2).tolist():
        if v > 0:
            reached = _dist_sq(r2 == v, math.isqrt(v)) <= v
            ball = torch.where(reached, torch.maximum(ball, torch.full_like(ball, v)), ball)
    dia = 2.0 * torch.sqrt(ball.to(torch.float64))
    offsets = [(z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1) if (z, y, x) != (0, 0, 0)]

    def moved(a, o, fill):
        for axis in range(3):
            if o[axis]:
                a = _shifted(a, axis, o[axis], fill)
        return a

    interior = ball > 0
    zero = ball == 0
    for o in offsets:
        interior = interior & ~moved(zero, o, False)
    total = torch.zeros_like(dia)
    count = torch.zeros_like(dia)
    kept = torch.where(interior, dia, 0.0)
    for o in offsets:
        total += moved(kept, o, 0.0)
        count += moved(interior.to(torch.float64), o, 0.0)
    surface = torch.where(count > 0, total / torch.clamp(count, min=1.0), dia)
    return torch.where(mask, torch.where(interior, dia, surface), 0.0), ball


def _stats_exact(values, scale, quantiles):
    raw = values[values > 0].to(torch.float64).cpu().numpy()
    v = raw * float(scale)
    n = int(v.size)
    mean = float(v.mean())
    sd = float(v.std(ddof=1)) if n > 1 else 0.0
    out = dict(count=n, mean=mean, standard_deviation=sd, maximum=float(v.max()), coefficient_of_variation=sd / mean,
               sum=float(v.sum()), sum_of_squares=float((v * v).sum()))
    if quantiles:
        q = np.quantile(v, [0.5, 0.1, 0.25, 0.75, 0.9])
        out.update(median=float(q[0]), percentile_10=float(q[1]), percentile_25=float(q[2]),
                   percentile_75=float(q[3]), percentile_90=float(q[4]), interquartile_range=float(q[3] - q[2]))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "edt"):  # batches take too long; the squared distances are whole numbers
        return None
    state = prepare(case, seed)
    if kind == "stats":
        return _stats_exact(state["values"], case["scale"], case["quantiles"])
    if kind == "volume":
        bone, roi = state["bone"] != 0, state["roi"] != 0
        both = bone & roi
        inside = roi.clone()
        for axis in range(3):
            inside = inside & _shifted(roi, axis, 1, False) & _shifted(roi, axis, -1, False)
        nb, nr, ne = int(both.sum()), int(roi.sum()), int((both & ~inside).sum())
        vv = case["spacing"] ** 3
        return [nb, nr, ne, nb * vv, nr * vv, nb / nr, ne / nb]
    if case["d"] * case["h"] * case["w"] > _EXACT_VOXELS:
        return None
    if kind == "lt":
        mask = state["volume"] != 0
        if case["phase"] == "background":
            mask = ~mask
        m, sq = _thickness_exact(mask)
        return dict(map=m, squared=sq) if case["squared"] else dict(map=m)
    bone, roi = torch.as_tensor(state["bone"]).cuda() != 0, torch.as_tensor(state["roi"]).cuda() != 0
    q = _wants_quantiles(case["mode"])
    mt, _ = _thickness_exact(bone & roi)
    ms, _ = _thickness_exact(roi & ~bone)
    out = dict(thickness=_stats_exact(mt, case["spacing"], q), spacing=_stats_exact(ms, case["spacing"], q))
    if case["maps"]:
        out["thickness_map"], out["spacing_map"] = mt, ms
    return out
