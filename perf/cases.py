"""The work that users of this framework have it do, as cases to be timed.

A scatter estimate of a TOF-PET study is one chain: images are prepared, the
list-mode events are histogrammed, the single scatter simulation (SSS) runs
(once per outer iteration, the step everything else serves), its sampled
sinogram is upsampled, scaled to the prompts on the tails, and injected back
into the events.  Each case is one of these calls through the package's
public entry points, at sizes of the package's own workloads (``workloads.py``,
``bench.py``, the tests) and on its scanner of 760 crystals x 80 rings or
reduced forms of it; ``draw`` spreads the same calls over their ranges.

``exact`` restates each computed result in FP64 torch, without the package.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from opensss_gb300 import DataReduction, Datafile, RayTracing3DTOFBatch, TofSSS, Utils, geometry, workloads
from opensss_gb300.BackProjection import fit_bins_device, fit_device
from opensss_gb300.batch import BatchSSS
from opensss_gb300.Interpolation import upsample_device
from opensss_gb300.TailsMask import tail_mask_device

LIGHT_CM_PER_PS = 299792458.0 * 1e-10
DEV = "cuda"
PHASE = 0.37  # ring rotation (crystals): keeps rays from lattice points off exact voxel corners


def listed():
    return [
        # one non-TOF scatter update of a small bed position, where launches and latency count
        dict(name="sss_nontof_small", kind="sss", n=40, nz=20, vox=1.0, radius=10.0, nru=8, ndu=32, bins=1, kahan=False),
        # the headline: one TOF scatter update, 64x64x48 at 6 mm, 16 rings x 48 crystals, 13 bins of 39 mm
        dict(name="sss_tof13", kind="sss", n=64, nz=48, vox=0.6, radius=10.0, nru=16, ndu=48, bins=13, kahan=False),
        # fine TOF bins (33 of 15 mm) on a wider body, ragged volume and sampling
        dict(name="sss_tof33_ragged", kind="sss", n=71, nz=45, vox=0.56, radius=11.3, nru=15, ndu=57, bins=33, kahan=False),
        # several bed positions of different sizes and bin counts planned once and run as one batch
        dict(name="batch_uneven", kind="batch", count=3, pick=11, lo=32, hi=60),
        # the sampled sinogram of the headline spread to the full sinogram, all bins summed
        dict(name="upsample_full", kind="upsample", nd=760, nr=80, nru=16, ndu=48, bins=13),
        # the tail mask of the full scanner, every sixth crystal
        dict(name="mask_full", kind="mask", nd=760, nr=80, af=6, n=64, nz=48, vox=0.6, radius=10.0, acf=0.0),
        # scale factors of 13 TOF bins in one pass
        dict(name="fit_tof13", kind="fit", nd=380, nr=16, af=4, bins=13, n=40, nz=26, span=0),
        # one bin's scale factor with span (length-weighted back-projection)
        dict(name="fit_span", kind="fit", nd=190, nr=40, af=3, bins=1, n=37, nz=26, span=7),
        # a whole list-mode acquisition into the demo's reduced sinogram (mash 2, span 19, 6 TOF bins)
        dict(name="histogram_50M", kind="histogram", events=50_000_000, mash=2, span=19, bins=6, flags=True),
        # scatter rates written back into the events, full angular sampling of a shorter frame
        dict(name="inject_20M", kind="inject", events=20_000_000, mash=2, span=19, bins=6),
        # a reconstructed map of 400x400x280 voxels cropped and resized to the simulation's voxels
        dict(name="prep_400", kind="prep", n0=400, n1=400, n2=280, crop=600.0, cropz=480.0, out=75, outz=48),
        # a few thousand rays through the batched tracer: the smallest call
        dict(name="raytrace_3k", kind="raytrace", rays=3001, n=64, nz=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sss", "sss", "sss33", "batch", "upsample", "mask", "fit", "fitspan", "histogram", "inject",
                       "prep", "raytrace"])
    if kind == "sss":
        n = rng.randint(32, 64)
        bins = rng.choice([1, 3, 5, 8, 13, 13, 21])
        return dict(kind="sss", n=n, nz=rng.randint(20, 48), vox=round(38.4 / n, 3), radius=round(rng.uniform(8, 12), 2),
                    nru=rng.randint(4, 16), ndu=rng.randint(20, 48), bins=bins,
                    kahan=bins > 1 and rng.random() < 0.25)
    if kind == "sss33":
        n = rng.randint(40, 71)
        return dict(kind="sss", n=n, nz=rng.randint(24, 44), vox=round(40.0 / n, 3), radius=round(rng.uniform(8, 16), 2),
                    nru=rng.randint(5, 11), ndu=rng.randint(24, 48), bins=33, kahan=False)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 4), pick=rng.randint(100, 10**6), lo=32, hi=48)
    if kind == "upsample":
        nd = 2 * rng.randint(95, 380)
        return dict(kind="upsample", nd=nd, nr=rng.randint(16, 80), nru=rng.randint(4, 16), ndu=rng.randint(16, 48),
                    bins=rng.choice([1, 13, 33]))
    if kind == "mask":
        return dict(kind="mask", nd=2 * rng.randint(95, 380), nr=rng.randint(10, 80), af=rng.randint(6, 9),
                    n=rng.randint(32, 96), nz=rng.randint(24, 64), vox=0.4, radius=round(rng.uniform(6, 12), 2),
                    acf=rng.choice([0.0, 0.0, 1.03]))
    if kind == "fit":
        return dict(kind="fit", nd=2 * rng.randint(60, 190), nr=rng.randint(8, 24), af=rng.randint(3, 6),
                    bins=rng.choice([1, 3, 6, 13]), n=rng.randint(24, 48), nz=rng.randint(16, 32), span=0)
    if kind == "fitspan":
        return dict(kind="fit", nd=2 * rng.randint(60, 100), nr=rng.choice([20, 30, 40]), af=rng.randint(3, 6), bins=1,
                    n=rng.randint(24, 48), nz=rng.randint(16, 32), span=rng.choice([5, 7]))
    if kind == "histogram":
        return dict(kind="histogram", events=_log(rng, 200_000, 50_000_000), mash=rng.choice([1, 2, 4]), span=19,
                    bins=rng.choice([1, 6]), flags=rng.random() < 0.7)
    if kind == "inject":
        return dict(kind="inject", events=_log(rng, 200_000, 20_000_000), mash=2, span=19, bins=rng.choice([1, 3, 6]))
    if kind == "prep":
        n = rng.randint(128, 400)
        return dict(kind="prep", n0=n, n1=n + rng.randint(-9, 9), n2=rng.randint(80, 280),
                    crop=round(1.6 * n * rng.choice([rng.uniform(0.6, 0.93), rng.uniform(1.07, 1.2)]), 1),
                    cropz=float(rng.randint(60, 148)), out=rng.randint(32, 96), outz=rng.randint(20, 64))
    return dict(kind="raytrace", rays=_log(rng, 300, 300_000), n=rng.randint(24, 96), nz=rng.randint(16, 64))


# ---------------------------------------------------------------- what a program has in hand


@functools.lru_cache(maxsize=8)
def _scanner(nd, nr, phase):
    return workloads.ring_scanner(nd, nr, radius_cm=41.0, ring_pitch_cm=25.6 / nr, phase=phase)


@functools.lru_cache(maxsize=8)
def _sinogram(nd, nr):
    lor, si, _ = geometry.SinogramCoordinates(1, 1, 1, 1, nd, nr, ID_Shidt=False)
    return lor, si


@functools.lru_cache(maxsize=8)
def _span(nr, span):
    return DataReduction.SinogramLUT(nr, span, nr - 1)


@functools.lru_cache(maxsize=8)
def _upsample_tables(nd, nr, nru, ndu):
    lor, si = _sinogram(nd, nr)
    return geometry.upsample_tables(lor, si, nru, ndu, "legpair")


@functools.lru_cache(maxsize=1)
def _attenuation_table():
    """[2000, 2]: energy in steps of 0.5 keV and water's attenuation as the
    Klein-Nishina cross section scaled to 0.096 / cm at 511 keV."""
    e = 0.5 * np.arange(1, 2001)
    a = e / 511.0
    kn = ((1 + a) / a**2 * (2 * (1 + a) / (1 + 2 * a) - np.log1p(2 * a) / a) + np.log1p(2 * a) / (2 * a)
          - (1 + 3 * a) / (1 + 2 * a) ** 2)
    return np.stack([e, 0.096 * kn / kn[1021]], axis=1)


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _tof(bins):
    """(TOF range, resolution) in ps of a bin count: 39 mm bins up to 13 of
    them, else 507 mm divided evenly; one bin is the non-TOF case."""
    if bins == 1:
        return 1000.0, 1.0e6
    width = 3.9 if bins <= 13 else 50.7 / bins
    return workloads.tof_bins(bins, width)[0], 214.0


def _phantom(n, nz, vox, radius, seed):
    """Activity (5% voxel noise, as a reconstructed map has) and attenuation on the GPU, and their bounds in cm."""
    act, mu, bounds = workloads.cylinder_phantom((n, n, nz), vox, seed % 100_000, radius_cm=radius)
    act = torch.from_numpy(act).to(DEV)
    act *= 1.0 + 0.05 * (2.0 * torch.rand(act.shape, device=DEV, generator=_generator(seed)) - 1.0)
    return act, torch.from_numpy(mu).to(DEV), bounds


def _engine(nru, ndu, bins, sc):
    rng, res = _tof(bins)
    return TofSSS(sc.geometry, sc.normals, sc.detector_size_mm, _attenuation_table(), 0.12, 435.0, nru, ndu, (2, 2, 2),
                  res, rng, bins, device=DEV)


def _batch_members(c):
    """The uneven batch's instances: sizes, sampling and bin counts of the package's generator, from c["pick"]."""
    r = np.random.default_rng(c["pick"])
    out = []
    for i in range(c["count"]):
        n = int(r.integers(c["lo"], c["hi"] + 1))
        out.append(dict(n=n, nz=int(r.integers(24, 41)), vox=40.0 / n, radius=float(r.uniform(8, 14)),
                        nru=int(r.integers(8, 17)), ndu=int(r.integers(24, 41)), bins=[13, 33, 1, 13][i % 4]))
    return out


def _fit_geometry(c):
    sc = _scanner(c["nd"], c["nr"], PHASE)
    lor, si = _sinogram(c["nd"], c["nr"])
    zr = float(sc.geometry[-1, 0, 2]) + 0.16
    bounds = np.array([-19.2, -19.2, -zr, 19.2, 19.2, zr])
    if c["span"]:
        index = _span(c["nr"], c["span"])[0]
        geom, _ = geometry.expandRings(sc.geometry, sc.normals)
        return geom, lor, index, index.shape[0], bounds
    return sc.geometry, lor, np.ascontiguousarray(si.T), c["nr"] ** 2, bounds


def _prep_window(c):
    return Utils.crop_window((c["n0"], c["n1"], c["n2"]), (1.6, 1.6, 2.0), (c["crop"], c["crop"], c["cropz"]))


def _events(n, header, seed):
    """Seeded event records of the 760 x 80 scanner, 24 bytes each: time, random and normalisation values, TOF, IDs."""
    g = _generator(seed)
    ev = torch.empty((n, 6), dtype=torch.int32, device=DEV)
    ev[:, 0] = torch.arange(n, device=DEV, dtype=torch.float64).mul_(600_000.0 / n).to(torch.int32)
    for k in (1, 2):
        ev[:, k] = torch.empty(n, device=DEV).uniform_(0.5, 2.0, generator=g).view(torch.int32)
    # TOF: the quantiles of a 400 ps Gaussian in random order (some outside the range, as many for every seed)
    q = (torch.randperm(n, device=DEV, generator=g).double() + 0.5) / n
    ev[:, 3] = (math.sqrt(2.0) * 400.0 * torch.special.erfinv(2.0 * q - 1.0)).float().view(torch.int32)
    for k in (4, 5):
        ev[:, k] = torch.randint(0, 760 * 80, (n,), device=DEV, generator=g, dtype=torch.int32)
    return ev.view(torch.uint8).reshape(-1)


def prepare(case, seed):
    c, g = case, _generator(seed)
    kind = c["kind"]
    if kind == "sss":
        act, mu, size = _phantom(c["n"], c["nz"], c["vox"], c["radius"], seed)
        eng = _engine(c["nru"], c["ndu"], c["bins"], _scanner(760, 80, PHASE))
        return dict(case=c, engine=eng, act=act, mu=mu, size=size)
    if kind == "batch":
        sc, jobs = _scanner(760, 80, PHASE), []
        for i, m in enumerate(_batch_members(c)):
            act, mu, size = _phantom(m["n"], m["nz"], m["vox"], m["radius"], seed + i)
            flat = [x.permute(2, 1, 0).contiguous().reshape(-1) for x in (act, mu)]
            jobs.append((_engine(m["nru"], m["ndu"], m["bins"], sc), *flat, size, tuple(act.shape)))
        return dict(case=c, plan=BatchSSS(jobs, workspace_bytes=8 << 30))
    if kind == "upsample":
        nl = c["nru"] * c["ndu"]
        sampled = torch.rand((c["bins"], nl, nl), device=DEV, generator=g)
        return dict(case=c, sampled=sampled, tables=_upsample_tables(c["nd"], c["nr"], c["nru"], c["ndu"]))
    if kind == "mask":
        # a patient off the centre, on a table
        r = np.random.default_rng(seed)
        _, mu, size = _phantom(c["n"], c["nz"], c["vox"], c["radius"] + r.uniform(0.0, 0.5), seed)
        mu = torch.roll(mu, tuple(int(v) for v in r.integers(-2, 3, size=2)), dims=(0, 1))
        mu *= 1.0 + 0.02 * torch.rand(mu.shape, device=DEV, generator=g)
        half, top = max(1, int(0.8 * c["radius"] / c["vox"])), c["n"] // 2 + int((c["radius"] + 1.5) / c["vox"])
        mu[c["n"] // 2 - half:c["n"] // 2 + half, min(top, c["n"] - 1)] = 0.05
        lor, si = _sinogram(c["nd"], c["nr"])
        return dict(case=c, mu=mu, size=size, geom=_scanner(c["nd"], c["nr"], PHASE).geometry, lor=lor, si=si)
    if kind == "fit":
        geom, lor, order, nsl, bounds = _fit_geometry(c)
        ncell = (c["nd"] + 1) * (c["nd"] // 2)
        scat = torch.rand((c["bins"], ncell, nsl), device=DEV, generator=g).add_(0.25)
        rnd = torch.full((ncell, nsl), 2.8, device=DEV)
        prompts = torch.poisson(28.0 * scat + rnd, generator=g)
        mask = (torch.rand((ncell, nsl), device=DEV, generator=g) < 0.7).to(torch.uint8)
        scat *= 1e-6  # probabilities, as the simulation gives them
        return dict(case=c, geom=geom, lor=lor, order=order, bounds=bounds, scat=scat, rnd=rnd, prompts=prompts, mask=mask,
                    cell=np.arange(ncell, dtype=np.int64) * nsl, ring=np.arange(nsl, dtype=np.int64))
    if kind in ("histogram", "inject"):
        flags = c.get("flags", True)
        header = workloads.listmode_header("case_df", c["events"], random_flag=True, normalization_flag=True)
        ev = _events(c["events"], header, seed)
        if not flags:  # no correction fields: 16-byte records
            header = workloads.listmode_header("case_df", c["events"], random_flag=False, normalization_flag=False)
            ev = ev.view(torch.int32).reshape(-1, 6)[:, [0, 3, 4, 5]].contiguous().view(torch.uint8).reshape(-1)
        lor, _ = _sinogram(760 // c["mash"], 80)
        lut = _span(80, c["span"])[2]
        s = dict(case=c, events=ev, header=header, lor=lor, lut=lut)
        if kind == "inject":
            s["nsl"] = int(lut.max()) + 1
            shape = (c["bins"], int(lor[:, :, 1].max()) + 1, int(lor[:, :, 0].max()) + 1, s["nsl"])
            s["scat"] = torch.rand(shape, device=DEV, generator=g)
            s["factor"] = np.random.default_rng(seed).uniform(0.5, 2.0, c["bins"]).astype(np.float32)
        return s
    if kind == "prep":
        img = torch.rand((c["n0"], c["n1"], c["n2"]), device=DEV, generator=g)
        img = -torch.log1p(-img)  # positive and skewed, as an activity map is
        return dict(case=c, img=img)
    if kind == "raytrace":
        h = torch.tensor([25.0, 25.0, 18.0], device=DEV, dtype=torch.float64)
        ends = torch.rand((c["rays"], 2, 3), device=DEV, dtype=torch.float64, generator=g)
        return dict(case=c, lines=((2 * ends - 1) * h).reshape(-1, 6))
    raise ValueError(kind)


# ---------------------------------------------------------------- one pass


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "sss":
        return s["engine"].run(s["act"], s["mu"], s["size"], kahan=c["kahan"])
    if kind == "batch":
        return s["plan"].run()
    if kind == "upsample":
        return upsample_device(s["sampled"], s["tables"], c["bins"], (c["nd"] + 1) * (c["nd"] // 2), c["nr"] ** 2)
    if kind == "mask":
        return tail_mask_device(s["mu"], s["size"], s["geom"], s["lor"], s["si"], c["af"],
                                acf_below=c["acf"] or None)
    if kind == "fit":
        a = (s["cell"], s["ring"], np.array([c["n"], c["n"], c["nz"]]), s["bounds"], s["geom"], s["lor"], s["order"],
             c["af"])
        if c["bins"] == 1:
            return np.array([fit_device(s["prompts"][0], s["rnd"], s["mask"], s["scat"][0], *a, span=c["span"] > 0)],
                            dtype=np.float32)
        return fit_bins_device(s["prompts"], s["rnd"], s["mask"], s["scat"], s["scat"][0].numel(), *a,
                               span=c["span"] > 0)
    if kind == "histogram":
        return Datafile.histogram_device(s["events"], s["header"], s["lor"], s["lut"], c["bins"], 1000.0, mash=c["mash"])
    if kind == "inject":
        return Datafile.inject_device(s["events"], s["header"], s["lor"], s["lut"], s["nsl"], s["scat"], s["factor"],
                                      1000.0, mash=c["mash"])
    if kind == "prep":
        return Utils.CropAndDownscale(s["img"], (1.6, 1.6, 2.0), (c["crop"], c["crop"], c["cropz"]),
                                      (c["out"], c["out"], c["outz"]))
    grid, bounds = _ray_grid(c)
    return RayTracing3DTOFBatch(grid, bounds, s["lines"], as_numpy=False)


def _ray_grid(c):
    return np.array([c["n"], c["n"], c["nz"]]), np.array([-19.2, -19.2, -14.4, 19.2, 19.2, 14.4])


# ---------------------------------------------------------------- what a pass cannot do without


def _sss_work(m):
    """Scatter points of the body x (ordered) leg pairs: the pair's factors
    once (~40 operations), and for the quarter of the pairs that pass the
    energy window each voxel of the leg once (weight, multiply, add)."""
    nl = m["nru"] * m["ndu"]
    area = math.pi * (m["radius"] / (2 * m["vox"])) ** 2
    points = area * min(18.0, m["nz"] * m["vox"]) / (2 * m["vox"])
    voxels = 1.3 * m["radius"] / m["vox"]
    per = 20.0 + (0.5 * voxels * 4.0 if m["bins"] > 1 else 0.0)
    nbytes = 8.0 * m["n"] ** 2 * m["nz"] + 4.0 * m["bins"] * nl * nl
    return nbytes, points * nl * nl * per


def work(case):
    c, kind = case, case["kind"]
    if kind == "sss":
        b, f = _sss_work(c)
        return {"bytes": b, "flops": f}
    if kind == "batch":
        each = [_sss_work(m) for m in _batch_members(c)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if kind == "upsample":
        nl = c["nru"] * c["ndu"]
        return {"bytes": 4.0 * ((c["nd"] + 1) * (c["nd"] // 2) * c["nr"] ** 2 + c["bins"] * nl * nl), "flops": 0.0}
    if kind == "mask":
        lors = math.ceil(c["nd"] / c["af"]) ** 2 / 2 * c["nr"] ** 2
        return {"bytes": (c["nd"] + 1) * (c["nd"] // 2) * c["nr"] ** 2 + 4.0 * c["n"] ** 2 * c["nz"],
                "flops": lors * 30.0}
    if kind == "fit":
        nsl = _fit_geometry(c)[3]
        lors = math.ceil(c["nd"] / c["af"]) ** 2 / 2 * nsl
        return {"bytes": lors * (5.0 + 8.0 * c["bins"]), "flops": lors * 0.5 * 1.3 * c["n"] * (2.0 * c["bins"] + 6.0)}
    if kind in ("histogram", "inject"):
        lor, _ = _sinogram(760 // c["mash"], 80)
        cells = (int(lor[:, :, 1].max()) + 1) * (int(lor[:, :, 0].max()) + 1) * (int(_span(80, c["span"])[2].max()) + 1)
        rec = 24.0 if c.get("flags", True) else 16.0
        if kind == "histogram":
            return {"bytes": c["events"] * rec + cells * (2.0 * c["bins"] + (8.0 if c["flags"] else 0.0)), "flops": 0.0}
        return {"bytes": c["events"] * (rec + 28.0 + 4.0), "flops": 0.0}
    if kind == "prep":
        w = _prep_window(c)
        inside = math.prod(max(0, min(x[2], n)) for x, n in zip(w, (c["n0"], c["n1"], c["n2"])))
        return {"bytes": 4.0 * (inside + c["out"] ** 2 * c["outz"]), "flops": 8.0 * inside}
    steps = 2 * c["n"] + c["nz"]
    return {"bytes": c["rays"] * (48.0 + 4.0 + 20.0 * steps), "flops": c["rays"] * 0.4 * steps * 12.0}


# ---------------------------------------------------------------- FP64 restatements


def _d(x):
    """A device scalar: torch divides by it, where a Python number would be multiplied by its rounded reciprocal."""
    return torch.tensor(float(x), dtype=torch.float64, device=DEV)


def _walk(lines, grid, bounds):
    """The voxels of every ray, one step at a time: yields (rays that have a
    voxel at this step, 1-based linear index, entry and exit parameters).  The
    Amanatides-Woo walk of the package's tracer in plain FP64 operations."""
    n = [int(v) for v in grid]
    b = [float(v) for v in bounds]
    s, e = lines[:, :3], lines[:, 3:]
    v = e - s
    tmin = torch.zeros_like(v[:, 0])
    hit = torch.ones_like(tmin, dtype=torch.bool)
    for k in range(3):
        inv = 1.0 / (v[:, k] + 1e-20)
        t0, t1 = (b[k] - s[:, k]) * inv, (b[3 + k] - s[:, k]) * inv
        lo, hi = torch.where(inv >= 0, t0, t1), torch.where(inv >= 0, t1, t0)
        if k == 0:
            tmin, tmax = lo, hi
            continue
        hit &= ~((tmin > hi) | (lo > tmax))
        tmin, tmax = torch.where(lo > tmin, lo, tmin), torch.where(hi < tmax, hi, tmax)
    hit &= ~(((tmin >= 1) & (tmax >= 1)) | ((tmin <= 0) & (tmax <= 0)))
    tmin, tmax = tmin.clamp(min=0.0), tmax.clamp(max=1.0)
    pos, end, st, tn, td = [], [], [], [], []
    for k in range(3):
        vs = (b[3 + k] - b[k]) / n[k]
        vk = v[:, k]
        a, z = s[:, k] + vk * tmin, s[:, k] + vk * tmax
        x = torch.ceil((a - b[k]) / _d(vs)).clamp(1.0, float(n[k]))
        end.append(torch.ceil((z - b[k]) / _d(vs)).clamp(1.0, float(n[k])).long())
        step = torch.sign(vk).long()
        plane = torch.where(step > 0, b[k] + x * vs, b[k] + (x - 1.0) * vs)
        moving = step != 0
        safe = torch.where(moving, vk, torch.ones_like(vk))
        tn.append(torch.where(moving, tmin + (plane - a) / safe, tmax))
        td.append(torch.where(moving, vs / safe.abs(), tmax))
        pos.append(x.long())
        st.append(step)
    live, prev = hit.clone(), tmin.clone()
    for _ in range(sum(n)):
        lin = pos[0] + (pos[1] - 1) * n[1] + (pos[2] - 1) * n[1] * n[0]
        last = (pos[0] == end[0]) & (pos[1] == end[1]) & (pos[2] == end[2])
        xy = tn[0] < tn[1]
        a = torch.where(xy, tn[0], tn[1])
        pa = a < tn[2]
        t = torch.where(last, tmax, torch.where(pa, a, tn[2]))
        yield live, lin, prev, t, (v, tmin)
        go = live & ~last
        for k, sel in enumerate((pa & xy, pa & ~xy, ~pa)):
            sel = sel & go
            tn[k] = torch.where(sel, tn[k] + td[k], tn[k])
            pos[k] = pos[k] + torch.where(sel, st[k], torch.zeros_like(st[k]))
        prev = torch.where(go, t, prev)
        live = go
        if not bool(live.any()):
            return


def _length(v, t0, t1):
    d = [v[:, k] * t0 - v[:, k] * t1 for k in range(3)]
    return torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])


def _exact_sss(m, act, mu, size, chunk=3_000_000):
    """Watson's single scatter sum as the package's SSS defines it, in FP64:
    leg integrals and voxel lists by the walk, then for every walking leg the
    activity of all scatter points collected per (partner, TOF offset) and
    multiplied by the TOF table."""
    f64 = dict(dtype=torch.float64, device=DEV)
    n, nz, nru, ndu, nb = m["n"], m["nz"], m["nru"], m["ndu"], m["bins"]
    sc = _scanner(760, 80, PHASE)
    rings = np.floor(np.linspace(0, 79, nru) + 0.5).astype(int)
    dets = np.zeros(ndu, dtype=int)
    for i in range(1, ndu):
        dets[i] = int(np.floor(dets[i - 1] + 760 / ndu))
    nl = nru * ndu
    di, ri = np.divmod(np.arange(nl), nru)
    geom = torch.from_numpy(sc.geometry[rings[ri], dets[di]]).to(**f64)
    geom[:, 2] = torch.from_numpy(sc.geometry[rings[ri], 0, 2]).to(**f64)
    nrm = torch.from_numpy(sc.normals[rings[ri], dets[di]]).to(**f64)
    di_t, ri_t = torch.from_numpy(di).to(DEV), torch.from_numpy(ri).to(DEV)
    # scatter points, z-slice major
    radius, zvox = -size[0], (size[5] - size[2]) / nz
    zs, ys, xs = torch.nonzero((mu[::2, ::2, ::2] > 0).permute(2, 1, 0), as_tuple=True)
    pts = torch.stack([(2 * xs + 1).double() * 2 * radius / _d(n) - radius,
                       (2 * ys + 1).double() * 2 * radius / _d(n) - radius, zvox / 2 + float(size[2]) + (2 * zs).double() * zvox], dim=1)
    npt = len(pts)
    # legs
    actf = act.permute(2, 1, 0).reshape(-1).double()
    muf = mu.permute(2, 1, 0).reshape(-1).double()
    A = torch.zeros((npt, nl), **f64)
    M = torch.zeros((npt, nl), **f64)
    cnt = torch.zeros((npt, nl), dtype=torch.long, device=DEV)
    cap = 2 * n + nz
    val = torch.zeros((npt, nl, cap), **f64) if nb > 1 else None
    rho = torch.zeros((npt, nl, cap), **f64) if nb > 1 else None
    most = 0
    per = max(1, chunk // nl)
    vec = geom[None] - pts[:, None]
    sv = vec.square().sum(-1).sqrt()
    for p0 in range(0, npt, per):
        p1 = min(npt, p0 + per)
        lines = torch.cat([pts[p0:p1, None].expand(-1, nl, -1), geom[None].expand(p1 - p0, -1, -1)], -1).reshape(-1, 6)
        a_, m_ = A[p0:p1].view(-1), M[p0:p1].view(-1)
        c_ = cnt[p0:p1].view(-1)
        svf = sv[p0:p1].reshape(-1)
        for live, lin, t0, t1, (v, tmin) in _walk(lines, (n, n, nz), size):
            ln = torch.where(live, _length(v, t0, t1), torch.zeros_like(t0))
            at = torch.where(live, lin - 1, torch.zeros_like(lin))
            w = actf[at] * ln
            a_ += w
            m_ += muf[at] * ln
            if nb > 1:
                k = torch.nonzero(w)[:, 0]
                val[p0:p1].view(-1, cap)[k, c_[k]] = w[k]
                rho[p0:p1].view(-1, cap)[k, c_[k]] = ((t1 - tmin) * svf)[k] / _d(LIGHT_CM_PER_PS)
                c_[k] += 1
    if nb > 1:
        most = int(cnt.max())
        val, rho = val[:, :, :most].contiguous(), rho[:, :, :most].contiguous()
    del vec
    unit = (geom[None] - pts[:, None]) / sv[..., None]
    inc = (unit * nrm[None]).sum(-1).abs() / nrm.norm(dim=-1)[None] / sv.square()
    # tables
    att = torch.from_numpy(_attenuation_table()).to(**f64)
    wid = 511 * 0.12 / 2 / math.sqrt(math.log(2))
    eff = torch.tensor([0.5 * (1 - math.erf((435.0 - e) / wid)) for e in att[:, 0].tolist()], **f64)
    eff = eff * eff[1021]
    ratio_mu = att[:, 1] / att[1021, 1]
    rng, res = _tof(nb)
    off = torch.arange(-4000, 4001, **f64)
    shift = (torch.arange(1, nb + 1, **f64) - (nb + 1) / 2) * (2 * rng / nb)
    T = torch.exp(-((off[:, None] - shift[None]) ** 2) / (res**2 / 4 / math.log(2)))
    tot = T.sum(1, keepdim=True)
    T = torch.where(tot > 0, T / torch.where(tot > 0, tot, torch.ones_like(tot)), torch.zeros_like(T))
    gam = 511.0e3 * 1.6e-19 / (9.10938356e-31 * 299792458.0**2)
    ds = sc.detector_size_mm[0] * sc.detector_size_mm[1] * 1e-2
    geo = ds * ds / (4 * math.pi)
    M = torch.where(M > 745.13, torch.full_like(M, math.inf), M)
    nslice = int(zs.max()) + 1 if npt else 0
    out = torch.zeros((nb, nl, nl), **f64)
    lp = torch.arange(nl, device=DEV)
    for lw in range(nl):
        # partner entries: every other leg, the same crystal's twice (either order)
        same = (di_t == di_t[lw]) & (lp != lw)
        parts = torch.cat([lp[lp != lw], lp[same]])
        first = torch.cat([di_t[lp[lp != lw]] >= di_t[lw], torch.zeros(int(same.sum()), dtype=torch.bool, device=DEV)])
        q = (unit[:, lw, None] * unit[:, parts]).sum(-1).clamp(-1.0, 1.0)
        row = (torch.floor(511.0 / (2.0 + q) + 0.5) * 2 - 1).long()
        ef = eff[row]
        Aw, Ap = A[:, lw, None], A[:, parts]
        ok = torch.isfinite(M[:, lw, None]) & torch.isfinite(M[:, parts]) & ~((Aw == 0) & (Ap == 0)) & (ef != 0)
        k = torch.where(ok, torch.where((Aw != 0) & (Ap != 0), 2.0, 1.0).double(), torch.zeros_like(q))
        per_slice = torch.zeros((nslice, len(parts)), **f64).index_add_(0, zs, k)
        den = gam * (1 + q) + 1
        r = 1 / den
        kn = r * r * (r + den - (1 - q * q))
        c = geo * inc[:, lw, None] * inc[:, parts] * ef * kn
        c = c * torch.exp(-M[:, lw, None]) * torch.exp(-M[:, parts] * ratio_mu[row])
        c = torch.where(ok & (Aw != 0), c / per_slice[zs].clamp(min=1.0), torch.zeros_like(c))
        l1 = torch.where(first, torch.full_like(parts, lw), parts)
        l2 = torch.where(first, parts, torch.full_like(parts, lw))
        if nb == 1:
            res_b = (c * Aw).sum(0)[:, None]
        else:
            sig = torch.where(first, -1.0, 1.0).double()
            u = -sig * (sv[:, lw, None] - sv[:, parts]) / _d(LIGHT_CM_PER_PS) + 4000.5
            hist = torch.zeros(len(parts) * 8001, **f64)
            i, j = torch.nonzero(c, as_tuple=True)
            t = torch.floor(u[i, j, None] + sig[j, None] * rho[i, lw]).long()
            t = torch.where(t < 0, t + 8001, t)
            hist.scatter_add_(0, (t + j[:, None] * 8001).reshape(-1), (c[i, j, None] * val[i, lw]).reshape(-1))
            res_b = hist.view(len(parts), 8001) @ T
        out.view(nb, -1).index_add_(1, l1 * nl + l2, res_b.T.contiguous())
    return out


def _lors(c, geom, npair_rings, lor):
    """(line [k, 6], cell, slice) of every lattice LOR: crystals d1 <= d2 on the af lattice, ring pairs fastest."""
    d = torch.arange(0, c["nd"], c["af"], device=DEV)
    i1, i2 = torch.meshgrid(d, d, indexing="ij")
    keep = i1 <= i2
    d1, d2 = i1[keep], i2[keep]
    r1, r2, sl = npair_rings
    d1, d2 = d1.repeat_interleave(len(r1)), d2.repeat_interleave(len(r1))
    reps = len(d1) // len(r1)
    r1, r2, sl = r1.repeat(reps), r2.repeat(reps), sl.repeat(reps)
    keep = (d1 < d2) | (r1 != r2)
    d1, d2, r1, r2, sl = d1[keep], d2[keep], r1[keep], r2[keep], sl[keep]
    g = torch.from_numpy(np.ascontiguousarray(geom)).to(DEV)
    lines = torch.cat([g[r1, d1, :2], g[r1, 0, 2:], g[r2, d2, :2], g[r2, 0, 2:]], 1)
    lt = torch.from_numpy(lor.astype(np.int64)).to(DEV)
    cell = lt[d1, d2, 1] * (c["nd"] // 2) + lt[d1, d2, 0]
    return lines, cell, sl


def _exact_fit(c, s):
    geom, lor, order, nsl, bounds = _fit_geometry(c)
    nr, nb = geom.shape[0], c["bins"]
    if c["span"]:
        two = np.float32(2) * np.asarray(order, dtype=np.float32)
        pr = (torch.from_numpy(two[:, 0].astype(np.int64)).to(DEV), torch.from_numpy(two[:, 1].astype(np.int64)).to(DEV),
              torch.arange(nsl, device=DEV))
    else:
        r1, r2 = torch.meshgrid(torch.arange(nr, device=DEV), torch.arange(nr, device=DEV), indexing="ij")
        pr = (r1.reshape(-1), r2.reshape(-1), torch.from_numpy(order.astype(np.int64)).to(DEV).reshape(-1))
    lines, cell, sl = _lors(c, geom, pr, lor)
    at = cell * nsl + sl
    m = (s["mask"].reshape(-1)[at] >= 1).double()
    keep = m > 0
    lines, at = lines[keep], at[keep]
    P = s["prompts"].reshape(nb, -1)[:, at].double()
    S = s["scat"].reshape(nb, -1)[:, at].double()
    R = s["rnd"].reshape(-1)[at].double()
    grid = (c["n"], c["n"], c["nz"])
    nvox = c["n"] * c["n"] * c["nz"]
    count = torch.zeros(len(at), dtype=torch.float64, device=DEV)
    total = torch.zeros_like(count)
    for live, lin, t0, t1, (v, _) in _walk(lines, grid, bounds):
        count += live
        if c["span"]:
            total += torch.where(live, _length(v, t0, t1), torch.zeros_like(t0))
    cols = torch.cat([P - R[None], S, torch.ones_like(R)[None]])  # the scatter is positive: every bin uses every LOR
    img = torch.zeros((2 * nb + 1, nvox), dtype=torch.float64, device=DEV)
    for live, lin, t0, t1, (v, _) in _walk(lines, grid, bounds):
        i = torch.nonzero(live)[:, 0]
        w = _length(v, t0, t1)[i] / total[i] if c["span"] else 1.0 / count[i]
        x = cols[:, i] * w
        x[-1] = 1.0
        for k in range(len(x)):
            img[k].scatter_add_(0, lin[i] - 1, x[k])
    seen = img[-1] > 0
    sens = torch.where(seen, img[-1], torch.ones_like(img[-1]))
    T = torch.where(seen, img[:nb] / sens, torch.zeros_like(img[:nb])).clamp(min=0.0)
    X = torch.where(seen, img[nb:2 * nb] / sens, torch.zeros_like(img[:nb])) * 1e10
    return ((X * T).sum(1) / (X * X).sum(1) * 1e10).cpu().numpy()


def _exact_histogram(c, s):
    """Randoms and normalisation: the value of each cell's last event."""
    if not c["flags"]:
        return None
    ev = s["events"].view(torch.int32).reshape(-1, 6)
    lor = torch.from_numpy(s["lor"].astype(np.int64)).to(DEV)
    lut = torch.from_numpy(s["lut"].astype(np.int64)).to(DEV)
    nrad, nang, nsl = int(lor[..., 1].max()) + 1, int(lor[..., 0].max()) + 1, int(lut.max()) + 1
    last = torch.full((nrad * nang * nsl,), -1, dtype=torch.int64, device=DEV)
    for e0 in range(0, len(ev), 5_000_000):
        a, b = ev[e0:e0 + 5_000_000, 4].long(), ev[e0:e0 + 5_000_000, 5].long()
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        c1, c2 = lo % 760, hi % 760
        r1 = torch.where(c1 < c2, lo // 760, hi // 760)
        r2 = torch.where(c1 < c2, hi // 760, lo // 760)
        d1, d2 = torch.minimum(c1, c2) // c["mash"], torch.maximum(c1, c2) // c["mash"]
        ang, rad, sl = lor[d1, d2, 0], lor[d1, d2, 1], lut[r1, r2]
        ok = (ang >= 0) & (rad >= 0) & (sl >= 0)
        cell = ((rad * nang + ang) * nsl + sl)[ok]
        idx = torch.arange(e0, e0 + len(a), device=DEV)[ok]
        last.scatter_reduce_(0, cell, idx, "amax")
    seen = last >= 0
    w = ev[last.clamp(min=0)]
    rnd = torch.where(seen, (w[:, 0].double() * 600.0) / c["bins"], torch.zeros_like(last, dtype=torch.float64))
    nrm = torch.where(seen, w[:, 1].contiguous().view(torch.float32).double(), torch.ones_like(last, dtype=torch.float64))
    shape = (nrad, nang, nsl)
    return None, rnd.reshape(shape), nrm.reshape(shape)


def _spline_axis(x):
    """Cubic B-spline coefficients along axis 0 (gain 6, pole sqrt(3) - 2, mirror start)."""
    z = math.sqrt(3.0) - 2.0
    y = 6.0 * x
    n = len(y)
    k = min(n, 28)
    y[0] = (y[:k] * (z ** torch.arange(k, dtype=torch.float64, device=DEV)).view(-1, *([1] * (x.dim() - 1)))).sum(0)
    for i in range(1, n):
        y[i] += z * y[i - 1]
    y[n - 1] = z / (z * z - 1) * (z * y[n - 2] + y[n - 1])
    for i in range(n - 2, -1, -1):
        y[i] = z * (y[i + 1] - y[i])
    return y


def _exact_prep(c, s):
    """Crop window, Gaussian, cubic spline on 12 repeated edge samples, sampling and clipping, axis by axis."""
    x = s["img"].double()
    out = (c["out"], c["out"], c["outz"])
    for d, (start, before, ln) in enumerate(_prep_window(c)):
        i = torch.arange(ln, device=DEV) - before + start
        ok = (i >= 0) & (i < x.shape[d])
        y = x.index_select(d, i.clamp(0, x.shape[d] - 1))
        shape = [1, 1, 1]
        shape[d] = ln
        x = y * ok.view(shape).double()
    lo, hi = x.min(), x.max()
    for d in range(3):
        x = x.movedim(d, 0)
        n = len(x)
        sigma = max(0.0, (n / out[d] - 1) / 2)
        if sigma > 1e-15:
            r = int(4 * sigma + 0.5)
            w = np.exp(-0.5 / sigma**2 * np.arange(-r, r + 1) ** 2)
            w /= w.sum()
            y = torch.zeros_like(x)
            for k in range(-r, r + 1):
                y += w[k + r] * x[(torch.arange(n, device=DEV) + k).clamp(0, n - 1)]
            x = y
        p = _spline_axis(x[(torch.arange(n + 24, device=DEV) - 12).clamp(0, n - 1)].contiguous())
        o = (torch.arange(out[d], device=DEV, dtype=torch.float64) + 0.5) * (n / out[d]) - 0.5
        f = torch.floor(o)
        t, i0 = o - f, f.long() + 11
        ws = ((1 - t) ** 3 / 6, (3 * t**3 - 6 * t**2 + 4) / 6, (-3 * t**3 + 3 * t**2 + 3 * t + 1) / 6, t**3 / 6)
        x = sum(p[i0 + k] * ws[k].view(-1, 1, 1) for k in range(4)).movedim(0, d)
    return x.clamp(lo, hi)


def _exact_raytrace(c, s):
    grid, bounds = _ray_grid(c)
    cap = int(grid.sum())
    k = len(s["lines"])
    lens = torch.zeros((k, cap), dtype=torch.float64, device=DEV)
    samples = torch.zeros_like(lens)
    run_sum = torch.zeros(k, dtype=torch.float64, device=DEV)
    for j, (live, lin, t0, t1, (v, _)) in enumerate(_walk(s["lines"], grid, bounds)):
        d = torch.where(live, _length(v, t0, t1), torch.zeros_like(t0))
        run_sum = run_sum + d / 2
        lens[:, j] = d
        samples[:, j] = torch.where(live, run_sum, torch.zeros_like(d))
    return None, lens, None, samples


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "sss":
        act, mu, size = _phantom(c["n"], c["nz"], c["vox"], c["radius"], seed)
        return _exact_sss(c, act, mu, size)
    if kind == "batch":
        out = []
        for i, m in enumerate(_batch_members(c)):
            out.append(_exact_sss(m, *_phantom(m["n"], m["nz"], m["vox"], m["radius"], seed + i)))
        return out
    if kind == "mask":
        return None
    if kind == "inject":
        return None
    s = prepare(case, seed)
    if kind == "upsample":
        t = s["tables"]
        x = s["sampled"].double().clamp(min=0.0).sum(0).reshape(-1)
        cell, ring = (torch.from_numpy(np.asarray(a)).to(DEV) for a in t[:2])
        return x[cell[:, None] + ring[None, :]]
    if kind == "fit":
        return _exact_fit(c, s)
    if kind == "histogram":
        return _exact_histogram(c, s)
    if kind == "prep":
        return _exact_prep(c, s)
    return _exact_raytrace(c, s)
