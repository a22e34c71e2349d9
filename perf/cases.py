"""The imaging work that users of sde_gb300 time: jobs, major cycles, CLEANs, mosaics, model
prediction, direct transforms and the Fortran drop-ins, each through its public entry point.

Observations are Earth-rotation tracks of a Y array (27 to 64 antennas), channel-major, with
weights that vary by visibility, one visibility in a hundred flagged, a power-law point sky
and noise; array and cell size are matched so that the longest baselines reach 0.94 of the
half grid (about two pixels per beam), as an observer chooses them.  exact() restates each
path in 64 bits with torch alone.
"""
import ctypes as C
import math

import numpy as np
import torch

from sde_gb300 import _abi, imaging, serve
from sde_gb300._abi import lib
from sde_gb300.mosaic import Mosaic

DEC = 40.0
N_SRC = 10


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # one integration of a 27-antenna array, imaged as it arrives: the served job's latency
        {"name": "job_snapshot_256", "kind": "job", "ants": 27, "ints": 1, "chans": 1, "imsize": 256,
         "rmode": "NORM", "robust": 0.0},
        # an ordinary single-channel synthesis, 8 h at 120 s: uniform weights, PSF, dirty image
        {"name": "uvmap_84k_512", "kind": "uvmap", "ants": 27, "ints": 240, "chans": 1, "imsize": 512,
         "rmode": "NONE", "robust": 0.0},
        # the large single field, 8 h at 10 s x 64 channels: robust weights, PSF, dirty image
        {"name": "uvmap_65m_4096", "kind": "uvmap", "ants": 27, "ints": 2880, "chans": 64, "imsize": 4096,
         "rmode": "NORM", "robust": 0.0},
        # CLEAN major cycle (model out of the residual, residual imaged) of the ordinary field
        {"name": "cycle_84k_512", "kind": "cycle", "ants": 27, "ints": 240, "chans": 1, "imsize": 512},
        # and of the large one: the headline step
        {"name": "cycle_65m_4096", "kind": "cycle", "ants": 27, "ints": 2880, "chans": 64, "imsize": 4096},
        # Hogbom minor cycles: the ordinary field's window, many components ...
        {"name": "hogbom_255_1000", "kind": "hogbom", "imsize": 512, "niter": 1000, "gain": 0.1},
        # ... and the large field's window, one major cycle's worth
        {"name": "hogbom_2047_200", "kind": "hogbom", "imsize": 4096, "niter": 200, "gain": 0.1},
        # Clark CLEAN, the clean task's default: transfer function, list, minor cycle, residual
        {"name": "clark_2048_300", "kind": "clark", "imsize": 2048, "niter": 300, "gain": 0.1, "flux": 0.2},
        # a mosaic of 49 uneven pointings, re-imaged each major cycle
        {"name": "mosaic_49", "kind": "mosaic", "points": 49, "vis_lo": 2000, "vis_hi": 2000000,
         "size_lo": 256, "size_hi": 2048},
        # model prediction (vismodel's padded degrid) for 16 channels from an odd-sized image
        {"name": "predict_1m3_1499", "kind": "predict", "ants": 27, "ints": 240, "chans": 16, "imsize": 1499},
        # uvmap's and vismodel's direct-transform options on a small ragged image
        {"name": "dft_84k_300", "kind": "dft", "ants": 27, "ints": 240, "chans": 1, "nx": 300, "ny": 277},
        # a Fortran program's major cycle through the drop-ins, on its own pageable arrays
        {"name": "dropin_1m3_1024", "kind": "dropin", "ants": 27, "ints": 240, "chans": 16, "imsize": 1024},
    ]


def _logi(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _obs_draw(rng, most):
    """ants, ints, chans with ants*(ants-1)/2*ints*chans spread over its logarithm up to most."""
    ants = rng.randint(27, 64)
    nbl = ants * (ants - 1) // 2
    rows = max(1, _logi(rng, nbl, most) // nbl)
    chans = min(64, _logi(rng, 1, rows))
    return {"ants": ants, "ints": max(1, rows // chans), "chans": chans}


def _size(rng, lo, hi):
    """An image size: a power of two half of the time, else any, odd ones among them."""
    if rng.random() < 0.5:
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    return _logi(rng, lo, hi)


def draw(rng):
    kind = rng.choice(["job", "uvmap", "uvmap", "cycle", "cycle", "hogbom", "hogbom", "clark", "mosaic",
                       "predict", "dft", "dropin"])
    rmode = rng.choice(["NORM", "NONE", "NATURAL"])
    robust = round(rng.uniform(-2.0, 2.0), 3)
    if kind == "job":
        ants = rng.randint(27, 64)
        return {"kind": kind, "ants": ants, "ints": rng.randint(1, 60), "chans": _logi(rng, 1, 64),
                "imsize": _size(rng, 256, 4096), "rmode": rng.choice(["NORM", "NATURAL"]), "robust": robust}
    if kind == "uvmap":
        return {"kind": kind, **_obs_draw(rng, 3e7), "imsize": _size(rng, 256, 4096), "rmode": rmode,
                "robust": robust}
    if kind == "cycle":
        return {"kind": kind, **_obs_draw(rng, 5e7), "imsize": _size(rng, 256, 4096)}
    if kind == "hogbom":
        n = _size(rng, 256, 4096)
        return {"kind": kind, "imsize": n, "niter": _logi(rng, 100, 1000 if n <= 1024 else 300),
                "gain": rng.choice([0.1, 0.05, 0.2])}
    if kind == "clark":
        return {"kind": kind, "imsize": 2 ** rng.randint(8, 12), "niter": _logi(rng, 50, 400), "gain": 0.1,
                "flux": 0.2}
    if kind == "mosaic":
        return {"kind": kind, "points": rng.randint(7, 49), "vis_lo": 2000, "vis_hi": _logi(rng, 2e4, 2e6),
                "size_lo": 256, "size_hi": 2 ** rng.randint(9, 11)}
    if kind == "predict":
        return {"kind": kind, **_obs_draw(rng, 4e6), "imsize": _size(rng, 256, 2048)}
    if kind == "dft":
        nx, ny = rng.randint(64, 320), rng.randint(64, 280)
        return {"kind": kind, **_obs_draw(rng, 8e4), "nx": nx, "ny": ny}
    return {"kind": kind, **_obs_draw(rng, 1.3e6), "imsize": _size(rng, 256, 1024)}


def _nvis(c):
    return c["ants"] * (c["ants"] - 1) // 2 * c["ints"] * c["chans"]


def _fft_flops(n):
    """A real 2-D FFT of n x n."""
    return 2.5 * n * n * math.log2(float(n) * n)


def _pow2(n):
    return imaging.fftpwr2(n)


def work(c):
    """Bytes: each input read once, each output written once.  Flops: 49 taps of a complex
    multiply-add per gridded or degridded visibility, the FFTs, the CLEAN updates."""
    k = c["kind"]
    if k in ("job", "uvmap"):
        n, p = _nvis(c), c["imsize"] ** 2
        return {"bytes": 24.0 * n + (4.0 * p if k == "job" else 4.0 * n + 8.0 * p),
                "flops": 49 * 6.0 * n + 2 * _fft_flops(_pow2(c["imsize"]))}
    if k == "cycle":
        n, p = _nvis(c), c["imsize"] ** 2
        return {"bytes": 24.0 * n + 8.0 * p, "flops": 49 * 8.0 * n + 2 * _fft_flops(_pow2(c["imsize"]))}
    if k == "hogbom":
        w = c["imsize"] // 2 - 1
        return {"bytes": 12.0 * w * w + 4.0 * c["imsize"] ** 2, "flops": 3.0 * w * w * c["niter"]}
    if k == "clark":
        n = c["imsize"]
        return {"bytes": 8.0 * n * n + 2.0 * n * n, "flops": 3 * _fft_flops(n) + 3.0 * n * n}
    if k == "mosaic":
        pts = _pointing_sizes(c, 0)
        n = sum(a for a, _ in pts)
        p = sum(s * s for _, s in pts)
        return {"bytes": 24.0 * n + 8.0 * p, "flops": 49 * 4.0 * n + sum(_fft_flops(s) for _, s in pts)}
    if k == "predict":
        n, m = _nvis(c), c["imsize"]
        return {"bytes": 4.0 * m * m + 24.0 * n, "flops": 49 * 4.0 * n + _fft_flops(_pow2(2 * m))}
    if k == "dft":
        n, p = _nvis(c), c["nx"] * c["ny"]
        return {"bytes": 24.0 * n + 12.0 * p + 8.0 * n, "flops": 12.0 * n * p}
    n, p = _nvis(c), c["imsize"] ** 2
    return {"bytes": 32.0 * n + 8.0 * p, "flops": 49 * 8.0 * n + 2 * _fft_flops(_pow2(c["imsize"]))}


# ---- inputs ---------------------------------------------------------------------------------
_CTX = []


def _ctx():
    """The program's library context (one per process, on torch's current stream)."""
    if not _CTX:
        _CTX.append(imaging.Context(0))
    return _CTX[0]


def _tracks(ants, ints, chans, cell, seed, hours=8.0):
    """u, v, w (float32, device), ordered [channel][time][baseline], 1.2-1.6 GHz."""
    rng = np.random.default_rng(seed)
    az = np.deg2rad([0.0, 120.0, 240.0])[np.arange(ants) % 3]
    r = rng.uniform(0.02, 1.0, ants) ** 1.5 * (10500.0 / cell)
    e, n, up = r * np.sin(az), r * np.cos(az), rng.normal(0.0, 2.0, ants)
    i, j = np.triu_indices(ants, 1)
    e, n, up = e[j] - e[i], n[j] - n[i], up[j] - up[i]
    lat, d = math.radians(34.0784), math.radians(DEC)
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    X, Y, Z = t(-math.sin(lat) * n + math.cos(lat) * up), t(e), t(math.cos(lat) * n + math.sin(lat) * up)
    hours = min(hours, ints * 10.0 / 3600.0) if ints <= 60 else hours
    H = t(np.deg2rad(((np.arange(ints) + 0.5) / ints - 0.5) * hours * 15.0))[:, None]
    s, c = torch.sin(H), torch.cos(H)
    um = s * X + c * Y
    vm = -math.sin(d) * c * X + math.sin(d) * s * Y + math.cos(d) * Z
    wm = math.cos(d) * c * X - math.cos(d) * s * Y + math.sin(d) * Z
    lam = t((1.2e9 + (np.arange(chans) + 0.5) * (0.4e9 / chans)) / 299792458.0)[:, None, None]
    return [(a[None] * lam).to(torch.float32).reshape(-1) for a in (um, vm, wm)]


def _sky(seed, half_rad, n=N_SRC):
    rng = np.random.default_rng(seed + 1)
    a = -1.5
    s = (0.02 ** a + rng.uniform(0, 1, n) * (1.0 - 0.02 ** a)) ** (1.0 / a)
    return s, rng.uniform(-half_rad, half_rad, n), rng.uniform(-half_rad, half_rad, n)


def _visibilities(u, v, sky, seed, noise=1e-3):
    out = torch.empty(u.numel(), dtype=torch.complex64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed + 2)
    for a in range(0, u.numel(), 1 << 23):
        uu, vv = u[a:a + (1 << 23)].double(), v[a:a + (1 << 23)].double()
        re, im = torch.zeros_like(uu), torch.zeros_like(uu)
        for s, l, m in zip(*sky):
            turns = uu * l + vv * m
            ph = (turns - torch.round(turns)).float() * (2.0 * math.pi)
            re += s * torch.cos(ph)
            im += s * torch.sin(ph)
        z = torch.complex(re.float(), im.float())
        out[a:a + (1 << 23)] = z + noise * torch.randn(z.numel(), dtype=torch.complex64, device="cuda", generator=g)
    return out


def _cell(imsize):
    """0.5 arcsec at 4096 pixels and coarser for smaller images, as fields of view go."""
    return 0.5 if imsize > 2048 else 1.0 if imsize > 512 else 2.0


def _observe(c, seed, imsize):
    cell = _cell(imsize)
    u, v, w = _tracks(c["ants"], c["ints"], c["chans"], cell, seed)
    half = 0.4 * imsize * math.radians(cell / 3600.0) * 0.5
    vis = _visibilities(u, v, _sky(seed, half), seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 3)
    wt = torch.rand(u.numel(), device="cuda", generator=g) + 0.5
    wt[torch.rand(u.numel(), device="cuda", generator=g) < 0.01] = -1.0
    return {"u": u, "v": v, "w": w, "vis": vis, "wt": wt, "cell": cell}


def _model_image(geom, seed, scale=0.6):
    """CLEAN components of the sky found so far: point pixels."""
    half = 0.4 * geom.nx * math.radians(geom.cellsize / 3600.0) * 0.5
    s, l, m = _sky(seed, half)
    cell = math.radians(geom.cellsize / 3600.0)
    img = torch.zeros((geom.ny, geom.nx), device="cuda")
    for f, a, b in zip(s, l, m):
        img[int(geom.ceny) - 1 + int(round(b / cell)), int(geom.cenx) - 1 - int(round(a / cell))] += scale * f
    return img


def _clean_images(n, seed):
    """PSF and dirty image (n x n, float32) of a tapered, uniformly weighted synthesis: the
    sampled cells of the uv plane, transformed; the sky convolved with that PSF, and noise."""
    u, v, _ = _tracks(27, 240, 16, _cell(n), seed)
    cu = 1.0 / (n * math.radians(_cell(n) / 3600.0))
    i, j = torch.round(u.double() / cu).long() % n, torch.round(v.double() / cu).long() % n
    hits = torch.bincount(torch.cat([j * n + i, ((-j) % n) * n + (-i) % n]), minlength=n * n)
    f = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    taper = torch.exp(-(f[:, None] ** 2 + f[None, :] ** 2) / (0.175 * n) ** 2)
    S = taper * hits.clamp(max=1).reshape(n, n)
    psf = torch.fft.ifft2(S).real
    rng = np.random.default_rng(seed + 5)
    sky = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for flux, x, y in zip(rng.uniform(0.1, 1.0, 60), rng.uniform(-0.2, 0.2, 60), rng.uniform(-0.2, 0.2, 60)):
        sky[int(round(y * n)) % n, int(round(x * n)) % n] += flux
    g = torch.Generator(device="cuda").manual_seed(seed + 4)
    noise = torch.fft.fft2(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))
    noise = torch.fft.ifft2(noise * torch.sqrt(S)).real
    dirty = torch.fft.ifft2(torch.fft.fft2(sky) * S).real / psf[0, 0] + noise * (2e-3 / noise.std())
    c = (n + 1) // 2 - 1  # uvmap's reference pixel
    place = lambda a: torch.roll(a, (c, c), (0, 1)).float().contiguous()  # noqa: E731
    return place(psf / psf[0, 0]), place(dirty)


def _pointing_sizes(c, seed):
    rng = np.random.default_rng(4000 + c["points"])
    n = np.exp(rng.uniform(math.log(c["vis_lo"]), math.log(c["vis_hi"]), c["points"])).astype(int)
    e = rng.integers(int(math.log2(c["size_lo"])), int(math.log2(c["size_hi"])) + 1, c["points"])
    return [(int(a), 2 ** int(b)) for a, b in zip(n, e)]


MOSAIC_CELL, MOSAIC_FWHM = 2.0, math.radians(0.5)


def _pointings(c, seed):
    side = int(math.ceil(math.sqrt(c["points"])))
    step = math.radians(0.25)
    out = []
    for k, (n, size) in enumerate(_pointing_sizes(c, seed)):
        u, v, w = (a[:n] for a in _tracks(27, -(-n // 351), 1, MOSAIC_CELL, seed + 10 * k))
        half = 0.4 * size * math.radians(MOSAIC_CELL / 3600.0) * 0.5
        vis = _visibilities(u, v, _sky(seed + k, half), seed + k)
        g = torch.Generator(device="cuda").manual_seed(seed + k)
        wt = torch.rand(n, device="cuda", generator=g) + 0.5
        row, col = divmod(k, side)
        out.append({"u": u, "v": v, "w": w, "vis": vis, "wt": wt, "imsize": size,
                    "l0": (col + 0.5 * (row % 2) - 0.5 * side) * step,
                    "m0": (row - 0.5 * side) * step * math.sqrt(3.0) / 2.0, "pb_fwhm_rad": MOSAIC_FWHM})
    return out


class _DevImage:
    """A library-owned device image as torch sees foreign memory; keeps its owner alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


def _batch_image(m, i, shape):
    p = C.c_void_p()
    _abi.check(lib().sde_batch_image(m.h, i, 0, C.byref(p)), "sde_batch_image")
    return torch.as_tensor(_DevImage(p.value, shape, m), device="cuda")


def prepare(c, seed):
    ctx, k = _ctx(), c["kind"]
    if k in ("job", "uvmap"):
        o = _observe(c, seed, c["imsize"])
        if k == "job":
            pin = {q: o[q].cpu().pin_memory() for q in ("u", "v", "w", "vis", "wt")}
            job = {"imsize": c["imsize"], "cell": o["cell"], "dec": DEC, "natural": c["rmode"] == "NATURAL",
                   "robust": c["robust"], "nvis": _nvis(c)}
            out = torch.empty((c["imsize"], c["imsize"]), dtype=torch.float32, pin_memory=True)
            return {"c": c, "ctx": ctx, "job": job, "pin": pin, "out": out}
        return {"c": c, "ctx": ctx, "o": o, "geom": imaging.Geom(c["imsize"], o["cell"], vdec=DEC)}
    if k == "cycle":
        o = _observe(c, seed, c["imsize"])
        geom = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
        ctx.weights(geom, o["u"], o["v"], o["w"], o["wt"], rmode="NORM")
        plan = imaging.Plan(ctx, geom, o["u"], o["v"], o["w"], o["vis"], o["wt"])
        psf, peak = ctx.image_buffer(geom), ctx.zeros(1, torch.float32)
        plan.image(psf, psf=True)
        ctx.image_max(psf, peak)
        cyc = imaging.MajorCycle(ctx, geom, plan, peak, psf)
        return {"c": c, "cycle": cyc, "model": _model_image(geom, seed)}
    if k == "hogbom":
        n = c["imsize"]
        psf, dirty = _clean_images(n, seed)
        lo, hi = imaging.Geom(n, _cell(n)).window()
        return {"c": c, "ctx": ctx, "psf": psf, "drt": dirty[lo:hi, lo:hi].contiguous()}
    if k == "clark":
        psf, dirty = _clean_images(c["imsize"], seed)
        return {"c": c, "ctx": ctx, "psf": psf, "dirty": dirty}
    if k == "mosaic":
        pts = [dict(p, **{q: p[q].cpu().numpy() for q in ("u", "v", "w", "vis", "wt")})
               for p in _pointings(c, seed)]
        m = Mosaic(ctx, pts, MOSAIC_CELL, rmode="UNIFORM")
        images = [_batch_image(m, i, (g.ny, g.nx)) for i, g in enumerate(m.geoms)]
        return {"c": c, "mosaic": m, "images": images,
                "sky": _batch_image(m, -1, (m.layout["mny"], m.layout["mnx"]))}
    if k == "predict":
        o = _observe(c, seed, c["imsize"])
        geom = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
        plan = imaging.Plan(ctx, imaging.padded_geom(geom), o["u"], o["v"], o["w"], o["vis"], o["wt"])
        return {"c": c, "ctx": ctx, "geom": geom, "plan": plan, "model": _model_image(geom, seed),
                "vis": torch.zeros_like(o["vis"]), "wt": o["wt"].clone()}
    if k == "dft":
        o = _observe(c, seed, max(c["nx"], c["ny"]))
        g = torch.Generator(device="cuda").manual_seed(seed + 6)
        image = torch.randn((c["ny"], c["nx"]), device="cuda", generator=g) * 0.01
        return {"c": c, "ctx": ctx, "o": o, "image": image, "vis": torch.zeros_like(o["vis"])}
    o = _observe(c, seed, c["imsize"])
    geom = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
    n, f32 = c["imsize"], np.float32
    h = {q: o[q].cpu().numpy() for q in ("u", "v", "w", "vis", "wt")}
    h.update(grid=np.zeros((geom.nv, geom.nu), np.complex64), dirty=np.zeros((n, n), f32),
             model=_model_image(geom, seed).cpu().numpy(), corrected=np.zeros((n, n), f32),
             mgrid=np.zeros((geom.nv, geom.nu), np.complex64), out=np.zeros(_nvis(c), np.complex64),
             cf=np.zeros(1 + 8 * 129, f32), ccf=np.zeros(1 + _pow2(n) // 2, f32),
             shift=np.ascontiguousarray(geom.shift, np.float64))
    lib().grdcf_(b"SF", _hp(h["cf"]), C.byref(C.c_int()), C.byref(C.c_int()), 2)
    lib().grdccf_(b"SF", _hp(h["ccf"]), _i(len(h["ccf"])), 2)
    return {"c": c, "geom": geom, "h": h}


# ---- one pass -------------------------------------------------------------------------------
def _hp(a):
    return a.ctypes.data_as(C.c_void_p)


def _i(x):
    return C.byref(C.c_int(int(x)))


def _f(x):
    return C.byref(C.c_float(float(x)))


def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "job":
        return serve.run_job(s["ctx"], s["job"], torch, s["pin"], s["out"])
    if k == "uvmap":
        o = s["o"]
        wt = o["wt"].clone()  # reweighted in place; the observation keeps its own
        r = imaging.uvmap(s["ctx"], s["geom"], o["u"], o["v"], o["w"], o["vis"], wt,
                          rmode="NORM" if c["rmode"] == "NATURAL" else c["rmode"], robust=(c["robust"], 0.0, 0.0),
                          weighting=c["rmode"] != "NATURAL")
        r["plan"].close()
        return {"dirty": r["dirty"], "psf": r["psf"], "peak": r["maxpsf"], "sumwt": r["sumwt"], "wt": wt}
    if k == "cycle":
        s["cycle"].degrid_step(s["model"])
        return s["cycle"].grid_step()
    if k == "hogbom":
        r = s["ctx"].hogbom(s["drt"], s["psf"], c["niter"], c["gain"])
        return {q: r[q] for q in ("cln", "res", "cflux", "cx", "cy", "ansub", "maxres", "tflux")}
    if k == "clark":
        r = imaging.clark(s["ctx"], s["dirty"], s["psf"], niter=c["niter"], gain=c["gain"], flux=c["flux"])
        return {q: r[q] for q in ("comp", "resid", "cl", "cx", "cy", "aniter", "tflux")}
    if k == "mosaic":
        s["mosaic"].dirty(graph=True)
        return {"mosaic": s["sky"], "images": s["images"]}
    if k == "predict":
        imaging.imgtovis(s["ctx"], s["geom"], s["plan"], s["model"], s["vis"], s["wt"])
        return {"vis": s["vis"], "wt": s["wt"]}
    if k == "dft":
        o, ctx = s["o"], s["ctx"]
        nx, ny = c["nx"], c["ny"]
        d = o["cell"] / 3600.0
        ax = ((nx + 1) // 2, -d, (ny + 1) // 2, d)
        r = imaging.dft_image(ctx, o["u"], o["v"], o["vis"], o["wt"], nx, ny, *ax)
        imaging.dft_vis(ctx, s["image"], *ax, o["u"], o["v"], o["wt"], s["vis"])
        return {"dirty": r["dirty"], "psf": r["psf"], "vis": s["vis"]}
    L, g, h = lib(), s["geom"], s["h"]
    n, nvis, sumwt = g.nx, len(h["wt"]), C.c_float()
    tabs = (_hp(h["cf"]), _i(3), _i(128), _hp(h["cf"]), _i(3), _i(128), _hp(h["shift"]))
    scal = (_i(nvis), _f(g.uscale), _f(0), _f(g.vscale), _f(0), _i(g.uorigin), _i(g.vorigin))
    fft = (_i(n), _i(n), _i(g.fnu), _i(g.nv))
    ccf = (_hp(h["ccf"]), _i(len(h["ccf"])), b"CORRECT")
    cen = (_f(g.cenx), _f(g.ceny), 7)
    L.grdh2d_(_hp(h["vis"]), _hp(h["wt"]), _hp(h["u"]), _hp(h["v"]), _hp(h["w"]), *scal, _hp(h["grid"]), _i(0),
              _i(g.nu), _i(g.nv), *tabs, C.byref(sumwt))
    L.fftr2d_(_hp(h["dirty"]), _hp(h["grid"]), None, None, None, *fft, _i(-1))
    L.pixcor2d_(_hp(h["dirty"]), _i(n), _i(n), *ccf, _hp(h["dirty"]), *cen)
    L.pixcor2d_(_hp(h["model"]), _i(n), _i(n), *ccf, _hp(h["corrected"]), *cen)
    L.fftr2d_(_hp(h["corrected"]), _hp(h["mgrid"]), None, None, None, *fft, _i(1))
    L.grddeh2d_(_hp(h["out"]), _hp(h["wt"]), _hp(h["u"]), _hp(h["v"]), _hp(h["w"]), *scal, _hp(h["mgrid"]),
                _i(g.nu), _i(g.nv), *tabs)
    return {"dirty": h["dirty"], "vis": h["out"], "wt": h["wt"], "sumwt": sumwt.value}


# ---- the same in 64 bits --------------------------------------------------------------------
SUPP, OSAMP = 3, 128


def _sf(nu):
    """The prolate spheroidal function psi(m=6, alpha=1) by Schwab's rational approximation."""
    nu = np.asarray(nu, np.float64)
    P = ((8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1),
         (4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2))
    Q = ((1.0, 8.212018e-1, 2.078043e-1), (1.0, 9.599102e-1, 2.918724e-1))
    f = []
    for p, q, end in zip(P, Q, (0.75, 1.0)):
        d = nu * nu - end * end
        f.append(sum(a * d ** i for i, a in enumerate(p)) / sum(a * d ** i for i, a in enumerate(q)))
    return np.where(nu < 0.75, f[0], np.where(nu <= 1.0, f[1], 0.0))


def _taps():
    """[129][7] tap weights by sub-cell offset (-64..64), from the REAL table of the gridder."""
    i = np.abs(np.arange(-(SUPP + 1) * OSAMP, (SUPP + 1) * OSAMP + 1)) / float(SUPP * OSAMP)
    cf = np.where(i <= 1.0, (1 - i * i) * _sf(np.minimum(i, 1.0)), 0.0).astype(np.float32)
    cf = cf / np.add.accumulate(cf)[-1]
    at = (SUPP + 1) * OSAMP + np.arange(-64, 65)[:, None] + OSAMP * np.arange(-SUPP, SUPP + 1)[None, :]
    return torch.as_tensor(cf[at].astype(np.float64), device="cuda")


def _nint(x):
    return torch.sign(x) * torch.floor(torch.abs(x) + 0.5)


def _cells(g, u, v, real):
    """1-based cells before the shift by SUPP, sub-cell offsets and the conjugation flag; real:
    in the 32-bit arithmetic that defines the degridder's and the weighting's cells."""
    f = torch.float32 if real else torch.float64
    cu = u.to(f) * float(g.uscale) if not real else u * torch.tensor(float(g.uscale), dtype=f, device="cuda")
    cv = v.to(f) * float(g.vscale) if not real else v * torch.tensor(float(g.vscale), dtype=f, device="cuda")
    conj = cu > 0
    sgn = torch.where(conj, 1.0, -1.0).to(f)
    cu, cv = sgn * cu + g.uorigin, sgn * cv + g.vorigin
    nu, nv = _nint(cu), _nint(cv)
    du, dv = _nint(OSAMP * (nu - cu)), _nint(OSAMP * (nv - cv))
    return nu.long(), nv.long(), du.long() + 64, dv.long() + 64, conj


def _weights64(g, u, v, wt, rmode, robust):
    nu, nv, _, _, _ = _cells(g, u, v, True)
    use = wt > 0
    on = use & (nu >= 1) & (nu <= g.nu) & (nv >= 1) & (nv <= g.nv)
    cell = torch.where(on, (nv - 1) * g.nu + nu - 1, 0)
    w = torch.where(on, wt.double(), 0.0)
    gwt = torch.zeros(g.nu * g.nv, dtype=torch.float64, device="cuda").index_add_(0, cell, w)
    f2, d2 = 1.0, 0.0
    if rmode == "NORM":
        f2, d2 = (5.0 * 10.0 ** -robust) ** 2 / float((gwt * gwt).sum() / w.sum()), 1.0
    half = torch.where((nu == g.uorigin) & (nv != g.vorigin), 0.5, 1.0)
    new = half * wt.double() / (gwt[cell] * f2 + d2)
    return torch.where(on, new, torch.where(use, -1.0, wt.double()))


def _grid64(g, u, v, vis, wt, psf=False):
    """The gridder's final half plane [nv][nu] (complex128) and the sum of the gridded weights."""
    taps = _taps()
    vis = None if psf else vis
    wide = g.nu + SUPP + 1
    raw = torch.zeros((g.nv * wide, 1 if psf else 2), dtype=torch.float64, device="cuda")
    lsum = swt = 0.0
    for a in range(0, u.numel(), 1 << 23):
        b = slice(a, a + (1 << 23))
        nu, nv, du, dv, conj = _cells(g, u[b], v[b], False)
        ok = (wt[b] > 0) & (nu + 2 * SUPP <= g.nu) & (nv + SUPP <= g.nv) & (nv - SUPP >= 1)
        nu, nv, du, dv, conj = (x[ok] for x in (nu, nv, du, dv, conj))
        w = wt[b][ok].double()
        tu, tv = taps[du], taps[dv]
        lsum += float((w * tu.sum(1) * tv.sum(1)).sum())
        swt += float(w.sum())
        if psf:
            val = w[:, None]
        else:
            z = vis[b][ok]
            val = torch.stack([w * z.real.double(), torch.where(conj, -w, w) * z.imag.double()], 1)
        for q in range(7):
            row = val * tv[:, q, None]
            at = (nv - 1 + q - SUPP) * wide + nu - 1
            for p in range(7):
                raw.index_add_(0, at + p, row * tu[:, p, None])
    raw = raw.reshape(g.nv, wide, -1)
    z = torch.complex(raw[..., 0], raw[..., 1]) if not psf else raw[..., 0].to(torch.complex128)
    # column UORIGIN + SUPP (0-based SUPP) is u = 0; fold the columns left of it and itself
    rows = torch.arange(g.nv, device="cuda")
    mirror = 2 * (g.vorigin - 1) - rows
    inside = (mirror >= 0) & (mirror < g.nv) & (torch.abs(rows - (g.vorigin - 1)) <= g.nv // 2 - 1)
    m = torch.where(inside, mirror, 0)
    z = z.clone()
    left = z[:, :SUPP + 1].clone()
    for k in range(SUPP + 1):
        z[:, SUPP + k] += torch.where(inside, left[m, SUPP - k].conj(), 0.0)
    out = torch.zeros((g.nv, g.nu), dtype=torch.complex128, device="cuda")
    out[:, :g.nu - SUPP] = z[:, SUPP:g.nu]
    return out * ((g.nu - 1) * float(g.nv) / lsum), swt


def _correction(g):
    f = lambda n, cen: torch.as_tensor(_sf(  # noqa: E731
        np.abs(np.round(2.0 * (_pow2(g.nx) // 2) / _pow2(n) * (np.arange(1, n + 1) - cen))) / (_pow2(g.nx) // 2)),
        device="cuda")
    return f(g.ny, g.ceny)[:, None] * f(g.nx, g.cenx)[None, :]


def _place(g):
    """Rows of the transform that the image's rows are, and likewise its columns."""
    cu, cv = (g.fnu + 1) // 2 - 1, (g.nv + 1) // 2 - 1
    y0 = (g.nv + 1) // 2 - (g.ny + 1) // 2
    rows = torch.arange(g.ny, device="cuda") + y0
    cols = (torch.arange(g.nx, device="cuda") + (g.fnu - g.nx) // 2 - cu) % g.fnu
    return rows, cols, cv


def _image64(g, grid, correct=True):
    rows, cols, cv = _place(g)
    x = torch.roll(torch.fft.ifft(torch.roll(grid, -cv, 0), dim=0), cv, 0)
    im = torch.fft.irfft(x, n=g.fnu, dim=1)[rows][:, cols]
    return im / _correction(g) if correct else im


def _model64(g, image, correct=True):
    rows, cols, cv = _place(g)
    full = torch.zeros((g.nv, g.fnu), dtype=torch.float64, device="cuda")
    full[rows[:, None], cols[None, :]] = image.double() / _correction(g) if correct else image.double()
    x = torch.fft.rfft(full, dim=1)
    return torch.roll(torch.fft.fft(torch.roll(x, -cv, 0), dim=0), cv, 0)


def _degrid64(g, grid, u, v, wt, old):
    """GRDDEH2D's visibilities: old where the weight is not positive."""
    taps, flat = _taps(), grid.reshape(-1)
    out = old.to(torch.complex128).clone()
    for a in range(0, u.numel(), 1 << 23):
        b = slice(a, a + (1 << 23))
        nu, nv, du, dv, conj = _cells(g, u[b], v[b], True)
        ok = (nu + SUPP <= g.nu) & (nv + SUPP <= g.nv) & (nv - SUPP >= 1)
        nu, nv = torch.where(ok, nu, 1 + SUPP), torch.where(ok, nv, 1 + SUPP)
        tu, tv = taps[du.clamp(0, 128)], taps[dv.clamp(0, 128)]
        acc = torch.zeros(nu.numel(), dtype=torch.complex128, device="cuda")
        for p in range(7):
            uc = nu - g.uorigin + p - SUPP
            neg = uc < 0
            for q in range(7):
                vc = nv - g.vorigin + q - SUPP
                row = (g.vorigin - 1 + torch.where(neg, -vc, vc)).clamp(0, g.nv - 1)
                z = flat[row * g.nu + torch.abs(uc)]
                acc += (tu[:, p] * tv[:, q]) * torch.where(neg, z.conj(), z)
        acc = acc / (tu.sum(1) * tv.sum(1))
        acc = torch.where(ok, torch.where(conj, acc.conj(), acc), 0.0)
        out[b] = torch.where(wt[b] > 0, acc, out[b])
    return out


def _hogbom64(drt, psf, niter, gain):
    res, p = drt.double().clone(), psf.double()
    ny, nx = res.shape
    pk = int(torch.argmax(torch.abs(p)))
    py, px = divmod(pk, p.shape[1])
    cln, cflux, tflux = torch.zeros_like(res), torch.zeros(niter, dtype=torch.float64, device="cuda"), 0.0
    flip = torch.flip(p, (0, 1))  # the beam index py + y - iy falls as iy rises
    for k in range(niter):
        at = int(torch.argmax(torch.abs(res)))
        y, x = divmod(at, nx)
        f = gain * float(res[y, x])
        tflux += f
        cln[y, x] += f
        cflux[k] = f
        res -= f * _window(flip, p.shape[0] - 1 - py - y, p.shape[1] - 1 - px - x, ny, nx)
    at = int(torch.argmax(torch.abs(res)))
    return cln, res, cflux, tflux, float(res.reshape(-1)[at])


def _window(a, y0, x0, ny, nx):
    out = torch.zeros((ny, nx), dtype=a.dtype, device=a.device)
    ya, yb, xa, xb = max(0, -y0), min(ny, a.shape[0] - y0), max(0, -x0), min(nx, a.shape[1] - x0)
    if yb > ya and xb > xa:
        out[ya:yb, xa:xb] = a[y0 + ya:y0 + yb, x0 + xa:x0 + xb]
    return out


def _clark64(dirty, psf, niter, gain, flux, numcl=32768, bpatch=128):
    """The first major cycle; None where the run goes on to a second."""
    n = dirty.shape[0]
    w, lo = n // 2, n // 4
    drt = dirty[lo:lo + w, lo:lo + w].double()
    p0 = max((n + 1) // 2 - bpatch // 2 + 1, 1) - 1
    p1 = min((n + 1) // 2 + bpatch // 2, n)
    patch = psf[p0:p1, p0:p1].double()
    out = torch.abs(psf).clone()
    out[p0:p1, p0:p1] = 0
    a = torch.abs(drt.float())
    amax, amin = float(a.max()), float(a.min())
    incr = np.float32(np.float32(amax) - np.float32(amin)) / np.float32(1023)
    index = torch.floor((a - amin) / torch.tensor(incr, device="cuda") + 0.5).long()
    hist = torch.bincount(index.reshape(-1).clamp(0, 1024), minlength=1025)[1:1025].cpu().numpy()
    tail = np.cumsum(hist[::-1])[::-1]
    full = np.nonzero(tail >= numcl)[0]
    slimi = int(full[-1]) + 2 if len(full) else 1
    slim = max(float(incr) * (slimi - 1) + amin + 0.5 * float(incr), float(out.max()) * amax)
    inlist = a > slim
    inlist &= torch.cumsum(inlist.reshape(-1), 0).reshape(w, w) <= numcl
    lst = torch.where(inlist, drt, 0.0)
    pk = int(torch.argmax(torch.abs(patch)))
    py, px = divmod(pk, patch.shape[1])
    flip = torch.flip(patch, (0, 1))
    comp, cl, tflux, smn, k = torch.zeros_like(drt), torch.zeros(niter, dtype=torch.float64, device="cuda"), 0.0, 0.0, 0
    for k in range(niter + 1):
        at = int(torch.argmax(torch.abs(lst)))
        y, x = divmod(at, w)
        top = float(lst[y, x])
        if k == niter:
            break
        smn += 1.0 / (k + 1)
        if abs(top) <= max(slim * smn, flux):
            if abs(top) > flux:
                return None
            break
        f = gain * top
        tflux += f
        cl[k] = f
        comp[y, x] += f
        beam = _window(flip, patch.shape[0] - 1 - py - y, patch.shape[1] - 1 - px - x, w, w)
        lst -= f * torch.where(inlist, beam, 0.0)
    g = imaging.Geom(n, 1.0)
    xfr = _model64(g, psf, correct=False)
    gw = _sub(g, w)
    resid = drt - _image64(gw, _model64(gw, comp, correct=False) * xfr, correct=False)
    return comp, resid, cl, tflux


class _sub:
    """A w x w image on geom's n x n transform."""

    def __init__(self, g, w):
        self.nx = self.ny = w
        self.fnu, self.nu, self.nv = g.fnu, g.nu, g.nv


def _uvmap64(g, o, rmode, robust):
    wt = o["wt"].double() if rmode == "NATURAL" else _weights64(g, o["u"], o["v"], o["wt"], rmode, robust)
    gp, swt = _grid64(g, o["u"], o["v"], None, wt, psf=True)
    psf = _image64(g, gp)
    gd, _ = _grid64(g, o["u"], o["v"], o["vis"], wt)
    return _image64(g, gd) / psf.max(), psf / psf.max(), psf.max().reshape(1), swt, wt


def exact(c, seed):
    k = c["kind"]
    if k in ("job", "uvmap"):
        o = _observe(c, seed, c["imsize"])
        g = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
        d, p, peak, swt, wt = _uvmap64(g, o, c["rmode"], c["robust"])
        return d if k == "job" else {"dirty": d, "psf": p, "peak": peak, "sumwt": swt, "wt": wt}
    if k == "cycle":
        o = _observe(c, seed, c["imsize"])
        g = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
        wt = _weights64(g, o["u"], o["v"], o["wt"], "NORM", 0.0)
        gp, _ = _grid64(g, o["u"], o["v"], None, wt, psf=True)
        peak = _image64(g, gp).max()
        m = _degrid64(g, _model64(g, _model_image(g, seed)), o["u"], o["v"], wt, o["vis"])
        gd, _ = _grid64(g, o["u"], o["v"], o["vis"].to(torch.complex128) - m, wt)
        return _image64(g, gd) / peak
    if k == "hogbom":
        psf, dirty = _clean_images(c["imsize"], seed)
        lo, hi = imaging.Geom(c["imsize"], _cell(c["imsize"])).window()
        cln, res, cflux, tflux, maxres = _hogbom64(dirty[lo:hi, lo:hi], psf, c["niter"], c["gain"])
        return {"cln": cln, "res": res, "cflux": cflux, "cx": None, "cy": None, "ansub": None,
                "maxres": maxres, "tflux": tflux}
    if k == "clark":
        psf, dirty = _clean_images(c["imsize"], seed)
        r = _clark64(dirty, psf, c["niter"], c["gain"], c["flux"])
        if r is None:
            return None
        return {"comp": r[0], "resid": r[1], "cl": r[2], "cx": None, "cy": None, "aniter": None, "tflux": r[3]}
    if k == "mosaic":
        return _mosaic64(c, seed)
    if k == "predict":
        o = _observe(c, seed, c["imsize"])
        g = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
        p = imaging.padded_geom(g)
        img = torch.zeros((p.ny, p.nx), dtype=torch.float64, device="cuda")
        y, x = int(p.ceny - g.ceny), int(p.cenx - g.cenx)
        img[y:y + g.ny, x:x + g.nx] = _model_image(g, seed)
        return {"vis": _degrid64(p, _model64(p, img), o["u"], o["v"], o["wt"], torch.zeros_like(o["vis"])),
                "wt": o["wt"].double()}
    if k == "dft":
        return _dft64(c, seed)
    o = _observe(c, seed, c["imsize"])
    g = imaging.Geom(c["imsize"], o["cell"], vdec=DEC)
    gd, swt = _grid64(g, o["u"], o["v"], o["vis"], o["wt"])
    vis = _degrid64(g, _model64(g, _model_image(g, seed)), o["u"], o["v"], o["wt"], torch.zeros_like(o["vis"]))
    return {"dirty": _image64(g, gd), "vis": vis, "wt": o["wt"].double(), "sumwt": swt}


def _mosaic64(c, seed):
    from sde_gb300.mosaic import mosaic_layout
    pts = _pointings(c, seed)
    mnx, mny, cx, cy, fw = mosaic_layout([(p["l0"], p["m0"]) for p in pts], [p["imsize"] for p in pts],
                                         math.radians(MOSAIC_CELL / 3600.0), MOSAIC_FWHM)
    num = torch.zeros((mny, mnx), dtype=torch.float64, device="cuda")
    den, images = torch.zeros_like(num), []
    for p, x, y, f in zip(pts, cx, cy, fw):
        g = imaging.Geom(p["imsize"], MOSAIC_CELL)
        im, _, _, _, wt = _uvmap64(g, p, "NONE", 0.0)
        images.append(im)
        n, cen = p["imsize"], (p["imsize"] + 1) // 2 - 1
        r = (torch.arange(n, device="cuda") - cen).double() ** 2
        pb = torch.exp(-4.0 * math.log(2.0) / float(f) ** 2 * (r[:, None] + r[None, :]))
        s = wt.clamp(min=0).sum()
        at = (slice(int(y) - 1 - cen, int(y) - 1 - cen + n), slice(int(x) - 1 - cen, int(x) - 1 - cen + n))
        num[at] += s * pb * im
        den[at] += s * pb * pb
    ok = den > 0.1 * den.max()
    return {"mosaic": torch.where(ok, num / torch.where(ok, den, 1.0), 0.0), "images": images}


def _dft64(c, seed):
    o = _observe(c, seed, max(c["nx"], c["ny"]))
    d = math.radians(o["cell"] / 3600.0)
    nx, ny = c["nx"], c["ny"]
    x = (torch.arange(1, nx + 1, device="cuda") - (nx + 1) // 2).double() * -d
    y = (torch.arange(1, ny + 1, device="cuda") - (ny + 1) // 2).double() * d
    g = torch.Generator(device="cuda").manual_seed(seed + 6)
    image = (torch.randn((ny, nx), device="cuda", generator=g) * 0.01).to(torch.complex128)
    w = o["wt"].double().clamp(min=0)
    w = w / w.sum()
    dirty = torch.zeros((ny, nx), dtype=torch.complex128, device="cuda")
    psf, vis = torch.zeros_like(dirty), []
    for a in range(0, w.numel(), 1 << 15):
        b = slice(a, a + (1 << 15))
        cis = lambda uv, ax: torch.exp(2j * math.pi * (uv[b].double()[:, None] * ax[None, :]))  # noqa: E731
        ex, ey = cis(o["u"], x), cis(o["v"], y)
        wb = w[b].to(torch.complex128)
        dirty += (ey.conj() * (wb * o["vis"][b])[:, None]).T @ ex.conj()
        psf += (ey.conj() * wb[:, None]).T @ ex.conj()
        vis.append(torch.where(w[b] > 0, ((ey @ image) * ex).sum(1), 0.0))
    return {"dirty": dirty.real, "psf": psf.real, "vis": torch.cat(vis)}
