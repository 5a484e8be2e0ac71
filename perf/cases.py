"""Workloads by which the library's speed is measured, through its public entry
points: bursts, scenes and stacks of synthetic Sentinel-1-like data.

``listed()`` names the fixed cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call (the
inputs, on the device or, for the drop-in, on the host; plans and output
buffers), ``run(state)`` makes one pass, ``work(case)`` counts the bytes and
operations the pass cannot do without, and ``exact(case, seed)`` computes the
pass's outputs in 64 bits with plain torch and numpy.

Data: circular complex Gaussian clutter with point targets 30 dB above it (the
backprojection), complex Gaussian echoes with a chirp's echoes among them (range
compression), partly coherent complex Gaussian images with an unformed (zero)
border (interferograms); volcano or sloped int16 DEMs.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from srg_b200 import _lib, api, scene

DEV = "cuda"
FS_MHZ = 64.345        # range sampling of the IW1 swath
RANFFT = 32768         # length of the reference's range-compression filter


# --------------------------------------------------------------------------
# the cases


def listed():
    return [
        # The smallest call: one tiny burst patch (the test suite's mini
        # scenes), as a quick look at a point or a unit test makes it; launch
        # and set-up latency decide.
        dict(name="bp_small", kind="bp", form="split", pulses=320, samples=384, width=48, length=40,
             spacing=2e-4, aperture=96, tops=True),
        # A burst over a small target area (configuration 0's sizes): fewer
        # tiles than the chip has room for.
        dict(name="bp_area", kind="bp", form="split", pulses=1024, samples=4096, width=256,
             length=256, spacing=2e-4, aperture=0, tops=False),
        # One IW1-sized burst onto its grid (configuration 1), device resident.
        dict(name="bp_iw1", kind="bp", form="split", pulses=1500, samples=21000, width=2400,
             length=1200, spacing=1e-4, aperture=0, tops=False),
        # The FP64 form, which a user takes for the reference's own arithmetic:
        # an odd-sized part of a burst.
        dict(name="bp_fp64", kind="bp", form="fp64", pulses=1321, samples=9001, width=917,
             length=601, spacing=1e-4, aperture=0, tops=False),
        # Finer interpolation (configuration 2): the burst's lines oversampled
        # 2x, then backprojected.
        dict(name="bp_oversampled", kind="bp2x", form="split", pulses=1500, samples=21000,
             width=2400, length=1200, spacing=1e-4, aperture=0, tops=False),
        # A full IW scene (configuration 3): 27 bursts in one plan, merged into
        # the scene raster.
        dict(name="scene_iw", kind="scene", swaths=3, bursts=9, scale=1.0),
        # One burst through the drop-in entry: pinned host lines, DEM and .geo
        # files, everything included.
        dict(name="dropin_iw1", kind="dropin", pulses=1500, samples=21000, width=2400, length=1200,
             spacing=1e-4, aperture=0, tops=False),
        # Range compression of one IW1 burst's decoded lines.
        dict(name="rc_iw1", kind="rc", lines=1500, samples=24000, pulse_us=52.4),
        # Range compression with a long pulse (more than 4,096 samples).
        dict(name="rc_long", kind="rc", lines=700, samples=29001, pulse_us=80.0),
        # Interferogram of a small ragged pair with looks (a quick look).
        dict(name="xm_small", kind="xm", images=2, width=917, length=601, looksac=4, looksdn=2),
        # The 31 sequential interferograms of a 32-pass stack (configuration 4),
        # single look.
        dict(name="xm_stack", kind="xm", images=32, width=2400, length=1200, looksac=1, looksdn=1),
        # Interferogram of two scene-wide images (the IW scene's raster), with
        # the looks that bring it to about 40 m.
        dict(name="xm_scene", kind="xm", images=2, width=16504, length=6646, looksac=4, looksdn=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bp", "bp", "fp64", "bp2x", "scene", "dropin", "rc", "rc", "xm", "xm", "xm"])
    if kind in ("bp", "fp64", "bp2x", "dropin"):
        pulses = _log(rng, 300, 1620)
        aperture = 0 if pulses >= 1000 else max(40, int(0.3 * pulses))
        big = kind in ("bp", "dropin")
        width, length = _log(rng, 40, 2600 if big else 1000), _log(rng, 40, 1300 if big else 600)
        spacing = rng.choice([1e-4, 2e-4]) if width < 600 else 1e-4
        samples = min(25600, int(3.2 * width * spacing / 1e-4) + _log(rng, 300, 12000))
        out = dict(kind="bp" if kind == "fp64" else kind, form="fp64" if kind == "fp64" else "split",
                   pulses=pulses, samples=samples, width=width, length=length, spacing=spacing,
                   aperture=aperture, tops=rng.random() < 0.3)
        if kind == "dropin":
            del out["form"]
        return out
    if kind == "scene":
        return dict(kind="scene", swaths=rng.randint(1, 3), bursts=rng.randint(1, 4),
                    scale=round(rng.uniform(0.3, 1.0), 3))
    if kind == "rc":
        pulse = round(rng.uniform(20.0, 60.0) if rng.random() < 0.75 else rng.uniform(64.0, 100.0), 2)
        return dict(kind="rc", lines=_log(rng, 8, 1500),
                    samples=rng.randint(int(pulse * FS_MHZ) + 500, RANFFT), pulse_us=pulse)
    width = _log(rng, 70, 16504)
    images = rng.choice([2, 2, 2, 3, 5, 8])
    length = _log(rng, 30, max(31, min(6646, int(1.0e8 / width / images))))
    looksac, looksdn = rng.choice([(1, 1), (1, 1), (2, 2), (4, 4), (5, 3), (10, 10), (3, 1)])
    return dict(kind="xm", images=images, width=width, length=length, looksac=looksac,
                looksdn=looksdn)


# --------------------------------------------------------------------------
# inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _clutter(shape, seed):
    z = torch.randn((*shape, 2), generator=_gen(seed), device=DEV)
    return torch.view_as_complex(z.mul_(math.sqrt(0.5)))


def _geometry(case, dem=None):
    """The burst's orbit, grid and scalars (a scene.Burst without samples)."""
    tops = dict(angc0=0.02, angc1=0.3) if case["tops"] else {}
    b = scene.make_geometry(pulses=case["pulses"], samples=2, width=case["width"],
                            length=case["length"], spacing=case["spacing"], centre_height=1000.0,
                            aperture=case["aperture"] or None, near_range=800.0e3, **tops)
    # the grid sits at the middle of the swath
    mid = 800.0e3 + 0.5 * (case["samples"] - 1) * b.dmrg
    b = scene.make_geometry(pulses=case["pulses"], samples=2, width=case["width"],
                            length=case["length"], spacing=case["spacing"], centre_height=1000.0,
                            aperture=b.aperture, near_range=mid, **tops)
    b.rngstart = 800.0e3
    b.rngend = b.rngstart + (case["samples"] - 1) * b.dmrg
    b.burst = np.zeros((0, case["samples"]), np.complex64)
    b.pulses = case["pulses"]
    return b


def _targets(b, dem, fl, lines, seed, count=200, amp=10.0 ** 1.5):
    """Adds the echoes of `count` point targets on random grid pixels (rows of
    `dem` from grid line fl) to the range lines, split over the two bins around
    each range; summed in a fixed order."""
    g = _gen(seed + 17)
    nl, W = dem.shape
    ll = torch.randint(0, nl, (count,), generator=g, device=DEV)
    pp = torch.randint(0, W, (count,), generator=g, device=DEV)
    x = _ecef(b, (ll + fl).double(), pp.double(), dem[ll, pp].double())
    s = torch.from_numpy(np.ascontiguousarray(b.satloc)).to(DEV)
    R = (x[:, None, :] - s[None]).square().sum(-1).sqrt()
    r = (R - b.rngstart) / b.dmrg
    i = r.floor()
    fr = r - i
    S = lines.shape[1]
    ok = (i >= 0) & (i + 1 < S)
    v = torch.polar(torch.full_like(R, amp), -4.0 * math.pi / b.wvl * R)
    k = torch.arange(R.shape[1], device=DEV)[None].expand_as(R)
    at = (k * S + i.clamp(0, S - 2).long())[ok]
    flat = torch.view_as_real(lines).view(-1, 2)
    for off, w in ((0, 1.0 - fr), (1, fr)):
        flat.index_put_((at + off,), torch.view_as_real(v * w)[ok].float(), accumulate=True)


def _dem(case, seed):
    L, W = case["length"], case["width"]
    if min(L, W) >= 64:
        return scene.volcano_dem_torch(seed, L, W, DEV, peak=1500.0, base=200.0)
    y = torch.arange(L, device=DEV)[:, None]
    x = torch.arange(W, device=DEV)[None]
    return (950 + 3 * x + 2 * y + torch.randint(-20, 21, (L, W), generator=_gen(seed), device=DEV)
            ).to(torch.int16)


def _burst_inputs(case, seed):
    """(Burst, DEM [length][width] int16, lines [P][S] complex64), on the device."""
    b = _geometry(case)
    dem = _dem(case, seed)
    lines = _clutter((case["pulses"], case["samples"]), seed + 1)
    _targets(b, dem, 0, lines, seed)
    return b, dem, lines


def _scene_inputs(case, seed):
    s = case["scale"]
    span = lambda lo, hi: (max(300, int(lo * s)), max(310, int(hi * s)))  # noqa: E731
    n = case["swaths"]
    grid, bursts = scene.iw_scene(
        seed=1003, nswaths=n, nbursts=case["bursts"],
        samples=tuple(int(v * s) for v in (18000, 21500, 25600))[:n], pulses=(1380, 1620),
        widths=span(2000, 2600), lengths=span(1000, 1300), dem_kind="flat")
    grid.dem = scene.volcano_dem_torch(seed, grid.length, grid.width, DEV, radius_frac=0.35)
    lines = []
    for i, b in enumerate(bursts):
        b.dem = grid.dem
        x = _clutter((b.rawdatalines, b.samples), seed * 100 + i)
        fl, ll, fp, lp = api.limits(b)
        _targets(b, grid.dem[fl:ll + 1], fl, x, seed * 100 + i)
        lines.append(x)
    return grid, bursts, lines


def _chirp(pulse_us):
    return dict(samplefreq=FS_MHZ, startfreq=-20.2, ramprate=40.8 / pulse_us, pulselength=pulse_us)


def _replica64(pulse_us):
    """The chirp replica: its sample times are single precision by the format
    of the pulse parameters, its phase double."""
    p = _chirp(pulse_us)
    sf = np.float32(p["samplefreq"])
    npts = int(np.float32(p["pulselength"]) * sf)
    t = (np.arange(npts, dtype=np.float32) / sf).astype(np.float64)
    ph = (2 * np.pi * np.float64(np.float32(p["startfreq"])) * t
          + np.pi * np.float64(np.float32(p["ramprate"])) * t * t)
    c = np.cos(ph).astype(np.float32) / np.float32(npts)
    s = np.sin(ph).astype(np.float32) / np.float32(npts)
    return torch.from_numpy((c + 1j * s).astype(np.complex128)).to(DEV), npts


def _rc_inputs(case, seed):
    n, S = case["lines"], case["samples"]
    x = _clutter((n, S), seed)
    rep, npts = _replica64(case["pulse_us"])
    d = torch.randint(0, S - npts, (3,), generator=_gen(seed + 1), device=DEV).tolist()
    for at in d:  # the chirp's echo, in every line
        x[:, at:at + npts] += (10.0 * npts / 100.0) * rep.to(torch.complex64)
    return x


def _xm_inputs(case, seed):
    """Images of partial coherence; a border of about 3 % is unformed (zero)."""
    nl, na = case["length"], case["width"]
    common = _clutter((nl, na), seed)
    ramp = torch.linspace(0.0, 12.0, na, device=DEV)
    out = []
    for k in range(case["images"]):
        x = _clutter((nl, na), seed * 50 + k + 1)
        x.mul_(0.5).addcmul_(common, torch.polar(torch.ones_like(ramp), 0.2 * k * ramp)[None])
        e = max(1, na // 64)
        x[:, :e] = 0
        x[:, na - e:] = 0
        x[:max(1, nl // 64)] = 0
        out.append(x)
    return out


# --------------------------------------------------------------------------
# the passes

_FORM = {"split": _lib.FORM_SPLIT, "fp64": _lib.FORM_FP64}
_streams = {}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("bp", "bp2x"):
        b, dem, lines = _burst_inputs(case, seed)
        return dict(kind=kind, form=_FORM[case["form"]],
                    burst=api.to_device(b, burst_tensor=lines, dem_tensor=dem))
    if kind == "scene":
        grid, bursts, lines = _scene_inputs(case, seed)
        dbs = [api.to_device(b, burst_tensor=x, dem_tensor=grid.dem, narrow_out=True)
               for b, x in zip(bursts, lines)]
        raster = torch.zeros((grid.length, grid.width), dtype=torch.complex64, device=DEV)
        plan = api.Scene(dbs, raster=raster, tile_shear=1000)  # the geometric shear
        return dict(kind=kind, plan=plan, raster=raster)
    if kind == "dropin":
        b, dem, lines = _burst_inputs(case, seed)
        pinned = torch.empty(lines.shape, dtype=torch.complex64, pin_memory=True)
        pinned.copy_(lines)
        where = "/dev/shm" if os.path.isdir("/dev/shm") else None
        fdem, fout = (tempfile.TemporaryFile(dir=where) for _ in range(2))
        fdem.write(dem.cpu().numpy().tobytes())
        fdem.flush()
        fout.truncate(8 * case["width"] * case["length"])
        call = api.prepare_azimuth_compress(b, fout.fileno(), fdem.fileno(), burst=pinned.numpy())
        return dict(kind=kind, call=call, files=(fdem, fout), keep=pinned,
                    shape=(case["length"], case["width"]))
    if kind == "rc":
        x = _rc_inputs(case, seed)
        pulse = _chirp(case["pulse_us"])
        nvalid = case["samples"] - _replica64(case["pulse_us"])[1]
        out = torch.empty((case["lines"], nvalid), dtype=torch.complex64, device=DEV)
        return dict(kind=kind, lines=x, pulse=pulse, out=out)
    if kind == "xm":
        imgs = _xm_inputs(case, seed)
        shape = (case["length"] // case["looksdn"], case["width"] // case["looksac"])
        outs = tuple([torch.empty(shape, dtype=torch.complex64, device=DEV) for _ in imgs[1:]]
                     for _ in range(2))
        return dict(kind=kind, images=imgs, outs=outs, looks=(case["looksac"], case["looksdn"]))
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "bp":
        api.backproject([state["burst"]], form=state["form"], sync=False)
        return state["burst"].out
    if kind == "bp2x":
        fine = api.oversample2(state["burst"], sync=False)
        api.backproject([fine], form=state["form"], sync=False)
        return fine.burst, fine.out
    if kind == "scene":
        # plans replay their graph on a stream of their own
        cur = torch.cuda.current_stream()
        s = _streams.setdefault(cur.device, None) or torch.cuda.Stream()
        _streams[cur.device] = s
        s.wait_stream(cur)
        state["plan"].run(stream=s.cuda_stream)
        cur.wait_stream(s)
        return state["raster"]
    if kind == "dropin":
        state["call"]()
        return np.memmap(state["files"][1], dtype=np.complex64, mode="r", shape=state["shape"])
    if kind == "rc":
        return api.range_compress(state["lines"], out=state["out"], sync=False, **state["pulse"])
    imgs, (lac, ldn) = state["images"], state["looks"]
    if len(imgs) == 2:
        return api.crossmul(imgs[0], imgs[1], looksac=lac, looksdn=ldn, sync=False)
    return api.crossmul_stack(imgs, looksac=lac, looksdn=ldn, sync=False, outs=state["outs"])


# --------------------------------------------------------------------------
# what a pass cannot do without


def _burst_work(b, form_bytes_out):
    """(formed terms, bytes of the range bins they read) of one burst over
    terrain of 1,000 m."""
    fl, ll, fp, lp = api.limits(b)
    coef = _centres(b, None)
    step = max(1, (lp - fp) // 256)
    azs, aze = _windows(b, torch.from_numpy(coef), torch.arange(fp, min(lp, b.demwidth - 1) + 1, step))
    n = (aze - azs).clamp(min=0)
    terms = float(n.sum()) * step
    rows = torch.nonzero(n.sum(1) > 0).flatten()
    if not len(rows):
        return 0.0, 0.0
    ends = np.array([int(rows[0]) + fl, int(rows[-1]) + fl], float)
    y, x = np.meshgrid(ends, np.array([fp, min(lp, b.demwidth - 1)], float))
    p = scene.llh_to_ecef(b.firstlat + y * b.deltalat, b.firstlon + x * b.deltalon,
                          np.full_like(y, 1000.0)).reshape(-1, 3)
    R = np.sqrt(((p[:, None] - b.satloc[None]) ** 2).sum(-1)).min(1)
    bins = min(b.samples, (R.max() - R.min()) / b.dmrg + 32)
    return terms, 8.0 * b.rawdatalines * bins


def work(case):
    kind = case["kind"]
    if kind in ("bp", "bp2x", "dropin"):
        b = _geometry(case)
        terms, band = _burst_work(b, 8)
        nbytes = band + (8 + 2) * case["width"] * case["length"] + 24 * case["pulses"]
        flops = 29 * terms
        if kind == "bp2x":  # the lines read once, the finer lines written once
            nbytes = nbytes - band + 24 * case["pulses"] * case["samples"]
            flops += 24 * case["pulses"] * case["samples"]
        return {"bytes": nbytes, "flops": flops}
    if kind == "scene":
        s = case["scale"]
        span = lambda lo, hi: (max(300, int(lo * s)), max(310, int(hi * s)))  # noqa: E731
        n = case["swaths"]
        grid, bursts = scene.iw_scene(
            seed=1003, nswaths=n, nbursts=case["bursts"],
            samples=tuple(int(v * s) for v in (18000, 21500, 25600))[:n], pulses=(1380, 1620),
            widths=span(2000, 2600), lengths=span(1000, 1300), dem_kind="flat")
        nbytes, flops = 0.0, 0.0
        for b in bursts:
            terms, band = _burst_work(b, 8)
            fl, ll, fp, lp = api.limits(b)
            flops += 29 * terms
            nbytes += band + 10.0 * (ll - fl + 1) * (min(lp, b.demwidth - 1) - fp + 1)
        return {"bytes": nbytes, "flops": flops}
    if kind == "rc":
        npts = int(np.float32(case["pulse_us"]) * np.float32(FS_MHZ))
        n, S = case["lines"], case["samples"]
        return {"bytes": 8.0 * n * (2 * S - npts), "flops": n * S * (2 * 5 * math.log2(4 * npts) + 6.0)}
    n, nl, na = case["images"], case["length"], case["width"]
    outs = (nl // case["looksdn"]) * (na // case["looksac"])
    nnn = 1 << max(1, (na - 1).bit_length())
    return {"bytes": 8.0 * (n * nl * na + 2 * (n - 1) * outs),
            "flops": n * nl * 10.0 * nnn * math.log2(nnn) + (n - 1) * 30.0 * nl * na}


# --------------------------------------------------------------------------
# the outputs in 64 bits


def _ecef(b, line, pix, h):
    """WGS-84 ECEF of grid pixels (torch float64 tensors)."""
    lat = torch.deg2rad(b.firstlat + line * b.deltalat)
    lon = torch.deg2rad(b.firstlon + pix * b.deltalon)
    e2 = 0.0066943799901499996
    s, c = torch.sin(lat), torch.cos(lat)
    re = 6378137.0 / torch.sqrt(1.0 - e2 * s * s)
    return torch.stack([(re + h) * c * torch.cos(lon), (re + h) * c * torch.sin(lon),
                        (re * (1.0 - e2) + h) * s], -1)


def _hermite(b, t):
    """Position and velocity at times t ([n]) by the 4-point Hermite of the
    state vectors, window clamped."""
    dt = b.timeorbit[1] - b.timeorbit[0]
    s = np.clip(np.trunc((t - b.timeorbit[0]) / dt).astype(np.int64), 2, b.numstatevec - 2) - 2
    idx = s[:, None] + np.arange(4)
    ts, xs, vs = b.timeorbit[idx], b.xx[idx], b.vv[idx]
    h, hd, sm = np.ones_like(ts), np.zeros_like(ts), np.zeros_like(ts)
    d = t[:, None] - ts
    for i in range(4):
        for j in range(4):
            if j != i:
                w = ts[:, i] - ts[:, j]
                h[:, i] *= d[:, j] / w
                sm[:, i] += 1.0 / w
                q = np.ones(len(t))
                for k in range(4):
                    if k not in (i, j):
                        q *= d[:, k] / (ts[:, i] - ts[:, k])
                hd[:, i] += q / w
    f0, f1 = 1.0 - 2.0 * d * sm, d
    g1, g0 = h + 2.0 * d * hd, 2.0 * (f0 * hd - h * sm)
    x = ((xs * f0[..., None] + vs * f1[..., None]) * (h * h)[..., None]).sum(1)
    v = ((xs * g0[..., None] + vs * g1[..., None]) * h[..., None]).sum(1)
    return x, v


def _centres(b, dem):
    """[nlines][3] parabolas of the azimuth centre along each grid line: zero
    Doppler times of the line's first, middle and last pixel (dem None: 1,000 m)."""
    fl, ll, fp, lp = api.limits(b)
    nl = ll - fl + 1
    half = (lp - fp) // 2 - 1
    ys = []
    for s in range(3):
        pix = fp + s * half
        if fp <= pix <= lp and 0 <= pix < b.demwidth:
            h = np.full(nl, 1000.0) if dem is None else dem[fl:ll + 1, pix].cpu().numpy().astype(np.float64)
            g = _ecef(b, torch.arange(fl, ll + 1).double(), torch.full((nl,), float(pix), dtype=torch.float64),
                      torch.from_numpy(h)).numpy()
        else:
            g = np.zeros((nl, 3))
        t = np.full(nl, float(b.tmid))
        x, v = np.tile(b.xyz_mid, (nl, 1)), np.tile(b.vel_mid, (nl, 1))
        live = np.arange(nl)
        for _ in range(51):
            fn = ((g[live] - x[live]) * v[live]).sum(1)
            step = fn / -(v[live] ** 2).sum(1)
            t[live] -= step
            x[live], v[live] = _hermite(b, t[live])
            live = live[np.abs(step) >= 5.0e-9]
            if not len(live):
                break
        rng = np.sqrt(((g - x) ** 2).sum(1))
        u = g - b.xyz_mid
        u /= np.sqrt((u ** 2).sum(1))[:, None]
        fd = 2.0 / b.wvl * (u @ b.vel_mid)
        ve = math.sqrt(float(np.dot(b.vel_mid, b.vel_mid)))
        num = rng * b.wvl / 2.0 / ve / ve * fd - rng * b.angc0 * math.pi / 180.0 / ve
        den = 1.0 + rng * b.angc1 * math.pi / 180.0 / ve
        ys.append(np.trunc(num / den * b.prf + float(b.rawdatalines // 2)))
    y0, y1, y2 = ys
    c = np.stack([0.5 * (y0 + y2 - 2.0 * y1), 0.5 * (y2 - y0), y1], -1)
    c[-1] = 0.0
    return c


def _windows(b, coef, pix):
    """Pulse window [azs, aze) of each line (rows of coef) at the given pixels."""
    fl, ll, fp, lp = api.limits(b)
    q = ((pix - fp).float() / torch.tensor(float(lp - fp), device=pix.device)).double()
    arg = (q * 2.0 - 1.0)[None]
    fit = coef[:, :1] * arg * arg + coef[:, 1:2] * arg + coef[:, 2:3]
    ap2, P = b.aperture // 2, b.rawdatalines
    ok = (fit > ap2) & (fit < P - ap2) & (fit > 0)
    away = lambda v: torch.where(v >= 0, torch.floor(v + 0.5), torch.ceil(v - 0.5))  # noqa: E731
    azs = away(fit - ap2).clamp(min=0).long()
    aze = away(fit + ap2).clamp(max=P - 1).long()
    return torch.where(ok, azs, 0), torch.where(ok, aze, 0)


def _image64(b, dem, lines, dmrg=None):
    """The backprojected image [nlines][demwidth] complex128: for each formed
    pixel the mean over its window of the linearly interpolated line times
    exp(+j 4 pi R / lambda)."""
    fl, ll, fp, lp = api.limits(b)
    dmrg = dmrg or b.dmrg
    P, S = lines.shape
    rmax = b.rngend - dmrg
    pix = torch.arange(fp, min(lp, b.demwidth - 1) + 1, device=DEV)
    azs, aze = _windows(b, torch.from_numpy(_centres(b, dem)).to(DEV), pix)
    out = torch.zeros((ll - fl + 1, b.demwidth), dtype=torch.complex128, device=DEV)
    yy, xx = torch.nonzero(aze > azs, as_tuple=True)
    sat = torch.from_numpy(np.ascontiguousarray(b.satloc)).to(DEV)
    flat = lines.reshape(-1)
    k4pi = 4.0 * math.pi / b.wvl
    for i in range(0, len(yy), 1 << 18):
        y, x = yy[i:i + (1 << 18)], xx[i:i + (1 << 18)]
        px = pix[x]
        p = _ecef(b, (y + fl).double(), px.double(), dem[y + fl, px].double())
        a0, a1 = azs[y, x][:, None], aze[y, x][:, None]
        acc = torch.zeros(len(y), dtype=torch.complex128, device=DEV)
        k0, k1 = int(a0.min()), int(a1.max())
        for ka in range(k0, k1, 64):
            k = torch.arange(ka, min(ka + 64, k1), device=DEV)
            R = torch.zeros((len(y), len(k)), dtype=torch.float64, device=DEV)
            for c in range(3):
                R.add_((p[:, c, None] - sat[None, k, c]).square_())
            R.sqrt_()
            ok = (k[None] >= a0) & (k[None] < a1) & (R >= b.rngstart) & (R <= rmax)
            r = (R - b.rngstart) / dmrg
            j = r.floor().clamp_(0, S - 2)
            w = r.sub_(j)
            at = (k[None] * S).add(j.long())
            v0, v1 = flat[at].to(torch.complex128), flat[at + 1].to(torch.complex128)
            v = v0 + (v1 - v0) * w
            acc += torch.where(ok, v * torch.polar(torch.ones_like(R), R.mul_(k4pi)), 0).sum(1)
        out[y, px] = acc / (a1 - a0)[:, 0]
    return out


def _fine64(lines):
    """2x-oversampled lines: the samples, and between them the 8-tap
    Hann-windowed sinc (unit DC gain)."""
    x = torch.arange(4, dtype=torch.float64) + 0.5
    h = torch.sinc(x) * 0.5 * (1.0 + torch.cos(math.pi * x / 4.0))
    h = (h / (2.0 * h.sum())).tolist()
    P, S = lines.shape
    pad = torch.zeros((P, S + 8), dtype=torch.complex128, device=DEV)
    pad[:, 4:4 + S] = lines
    out = torch.empty((P, 2 * S - 1), dtype=torch.complex128, device=DEV)
    out[:, ::2] = pad[:, 4:4 + S]
    odd = torch.zeros((P, S - 1), dtype=torch.complex128, device=DEV)
    for t in range(4):
        odd += h[t] * (pad[:, 4 - t:3 - t + S] + pad[:, 5 + t:4 + t + S])
    out[:, 1::2] = odd
    return out


def _crossmul64(a, b, lac, ldn):
    nl, na = a.shape[0] // ldn * ldn, a.shape[1]
    ncol = na // lac
    nnn = 1 << max(1, (na - 1).bit_length())
    ig = torch.empty((nl // ldn, ncol), dtype=torch.complex128, device=DEV)
    am = torch.empty_like(ig)
    rows = max(1, (1 << 24) // nnn // ldn) * ldn

    def up(x):
        X = torch.fft.fft(x, n=nnn, dim=1)
        U = torch.zeros((x.shape[0], 2 * nnn), dtype=torch.complex128, device=DEV)
        U[:, :nnn // 2] = X[:, :nnn // 2]
        U[:, 2 * nnn - nnn // 2:] = X[:, nnn // 2:]
        return torch.fft.ifft(U, dim=1)[:, :2 * na]  # unnormalised / nnn / 2

    def looks(v):
        v = v.reshape(-1, ldn, v.shape[1]).sum(1)[:, :ncol * lac]
        return v.reshape(-1, ncol, lac).sum(2)

    for l in range(0, nl, rows):
        x, y = a[l:min(l + rows, nl)].to(torch.complex128), b[l:min(l + rows, nl)].to(torch.complex128)
        u, v = up(x), up(y)
        two = lambda z: z.reshape(z.shape[0], na, 2).sum(2)  # noqa: E731
        g = looks(two(u * v.conj()))
        p = [looks(two(z.abs().square())).sqrt() for z in (u, v)]
        keep = (looks(x).abs() > 1e-6) & (looks(y).abs() > 1e-6)
        o = slice(l // ldn, l // ldn + g.shape[0])
        ig[o] = torch.where(keep, g, 0)
        am[o] = torch.where(keep, torch.complex(p[0], p[1]), 0)
    return ig, am


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bp", "dropin"):
        b, dem, lines = _burst_inputs(case, seed)
        img = _image64(b, dem, lines)
        if kind == "bp":
            return img
        fl, ll, fp, lp = api.limits(b)
        full = torch.zeros((case["length"], case["width"]), dtype=torch.complex128, device=DEV)
        full[fl:ll + 1] = img
        return full.cpu().numpy()
    if kind == "bp2x":
        b, dem, lines = _burst_inputs(case, seed)
        fine = _fine64(lines)
        return fine, _image64(b, dem, fine, dmrg=b.dmrg / 2.0)
    if kind == "scene":
        grid, bursts, lines = _scene_inputs(case, seed)
        raster = torch.zeros((grid.length, grid.width), dtype=torch.complex128, device=DEV)
        for b, x in zip(bursts, lines):
            fl, ll, fp, lp = api.limits(b)
            img = _image64(b, grid.dem, x)
            raster[fl:ll + 1] = torch.where(img.real.abs() > 1e-18, img, raster[fl:ll + 1])
        return raster
    if kind == "rc":
        x = _rc_inputs(case, seed)
        rep, npts = _replica64(case["pulse_us"])
        ref = torch.fft.fft(rep, n=RANFFT).conj()
        nvalid = case["samples"] - npts
        out = torch.empty((case["lines"], nvalid), dtype=torch.complex128, device=DEV)
        for l in range(0, len(x), 256):
            X = torch.fft.fft(x[l:l + 256].to(torch.complex128), n=RANFFT, dim=1)
            out[l:l + 256] = torch.fft.ifft(X * ref, dim=1)[:, :nvalid] * RANFFT
        return out
    imgs = _xm_inputs(case, seed)
    got = [_crossmul64(a, b, case["looksac"], case["looksdn"]) for a, b in zip(imgs, imgs[1:])]
    if len(imgs) == 2:
        return got[0]
    return [g for g, _ in got], [a for _, a in got]
