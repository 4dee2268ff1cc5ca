"""The work this library is timed on: calls a user's program makes, at the sizes it makes them.

Each case names a `kind` (a public call, or two that go together) and its sizes.
Observations are Earth-rotation tracks of a jittered 27-antenna Y array, so that
sample density, baseline order and duplicates are those of real uv coverage.
`exact` restates the arithmetic in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "casa-rs_gb300"))

import casars_cuda as cc  # noqa: E402
from casars_cuda import autograd as ag  # noqa: E402

DEV = "cuda"
C_LIGHT = 299_792_458.0
F64, F32, C64, C128, U8 = (torch.float64, torch.float32, torch.complex64, torch.complex128,
                           torch.uint8)
BASELINES = 351          # 27 antennas
MAX_EXACT_TAPS = 6.0e8   # kernel taps exact() evaluates in a few seconds


# ---- cases -----------------------------------------------------------------------
def listed():
    return [
        # a quick look at one snapshot: launches and latency count
        {"name": "dirty_256", "kind": "dirty", "image": 256, "rows": 4001, "planes": 0,
         "smin": 0, "smax": 0},
        # one hour of a compact array, the ordinary continuum image
        {"name": "dirty_512", "kind": "dirty", "image": 512, "rows": 126360, "planes": 0,
         "smin": 0, "smax": 0},
        # a long track on a large image of ragged size and row count
        {"name": "dirty_3000", "kind": "dirty", "image": 3000, "rows": 5000001, "planes": 0,
         "smin": 0, "smax": 0},
        # a wide-field snapshot: W-projection with small kernels
        {"name": "dirty_w_256", "kind": "dirty", "image": 256, "rows": 4000, "planes": 16,
         "smin": 4, "smax": 12},
        # differentiable imaging: model to visibilities and the gradient back
        {"name": "pair_w_2048", "kind": "pair", "image": 2048, "rows": 2021760, "planes": 32,
         "smin": 0, "smax": 0},
        # the wide-field headline: plan, grid and degrid 128 planes of large kernels
        {"name": "plan_w_4096", "kind": "plan", "image": 4096, "rows": 5054400, "planes": 128,
         "smin": 8, "smax": 64},
        # one major cycle of CLEAN over a kept plan
        {"name": "refresh_w_2048", "kind": "refresh", "image": 2048, "rows": 10108800,
         "planes": 64, "smin": 0, "smax": 0},
        # a spectral cube weighted, gridded and degridded in one call
        {"name": "cube_1024", "kind": "cube", "image": 1024, "rows": 1263600, "channels": 256},
        # the major cycle of a cube CLEAN: every plane's residual image from its model
        {"name": "cube_refresh_1000", "kind": "cube_refresh", "image": 1000, "rows": 270001,
         "channels": 101},
        # the minor cycle of CLEAN
        {"name": "hogbom_2048", "kind": "hogbom", "image": 2048, "niter": 2000, "boxed": False},
        # Briggs weights of a continuum data set
        {"name": "briggs_2048", "kind": "weights", "image": 2048, "rows": 10108800,
         "mode": "briggs"},
        # MeasurementSet rows to Stokes I samples
        {"name": "rows_64x4", "kind": "rows", "rows": 1263600, "channels": 64, "corr": 4,
         "spectrum": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dirty", "dirty", "dirty_w", "pair", "plan", "refresh", "cube",
                       "cube_refresh", "hogbom", "weights", "rows"])
    image = 2 * _logint(rng, 60, 1024)
    if kind in ("dirty", "weights"):
        image = _logint(rng, 120, 3000)
        rows = _logint(rng, 1000, 5000000)
        if kind == "weights":
            return {"kind": kind, "image": image, "rows": rows,
                    "mode": rng.choice(["natural", "uniform", "briggs"])}
        return {"kind": kind, "image": image, "rows": rows, "planes": 0, "smin": 0, "smax": 0}
    if kind == "dirty_w":
        return {"kind": "dirty", "image": max(image, 256), "rows": _logint(rng, 1000, 1000000),
                "planes": rng.randrange(2, 65), "smin": rng.randrange(3, 7),
                "smax": rng.randrange(7, 13)}
    if kind == "pair":
        return {"kind": kind, "image": image, "rows": _logint(rng, 1000, 2000000),
                "planes": rng.choice([0, rng.randrange(2, 65)]), "smin": 0, "smax": 0}
    if kind == "plan":
        return {"kind": kind, "image": 2 * rng.randrange(600, 1500),
                "rows": _logint(rng, 10000, 3000000), "planes": rng.randrange(16, 129),
                "smin": rng.randrange(4, 12), "smax": rng.randrange(16, 50)}
    if kind == "refresh":
        return {"kind": kind, "image": image, "rows": _logint(rng, 10000, 10000000),
                "planes": rng.choice([0, rng.randrange(2, 65)]), "smin": 0, "smax": 0}
    if kind in ("cube", "cube_refresh"):
        return {"kind": kind, "image": 2 * _logint(rng, 64, 512), "rows": _logint(rng, 3000, 300000),
                "channels": rng.randrange(3, 97)}
    if kind == "hogbom":
        return {"kind": kind, "image": _logint(rng, 128, 2048), "niter": _logint(rng, 30, 2000),
                "boxed": rng.random() < 0.5}
    return {"kind": "rows", "rows": _logint(rng, 500, 300000), "channels": _logint(rng, 1, 128),
            "corr": rng.choice([2, 4]), "spectrum": rng.random() < 0.5}


# ---- inputs ----------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _radius(image):
    return 1000.0 if image <= 600 else 5000.0 if image <= 1500 else 21000.0


def _cell(image, f_hi=1.4e9):
    """A third of the synthesised beam of the longest baseline (with its jitter)."""
    return 1.0 / (3.0 * 1.8 * _radius(image) * f_hi / C_LIGHT)


def _tracks(rows, radius, g):
    """uvw in metres, time-major, for one source seen for at most 8 hours."""
    r = torch.rand(30, generator=g, device=DEV, dtype=F64)
    k = torch.arange(9, device=DEV, dtype=F64)
    e, n = [], []
    for arm in range(3):
        rad = 40.0 * (radius / 40.0) ** (k / 8.0) * (1.0 - 0.03 * r[9 * arm:9 * arm + 9])
        az = math.radians(120.0 * arm)
        e.append(rad * math.sin(az))
        n.append(rad * math.cos(az))
    e, n = torch.cat(e), torch.cat(n)
    lat = math.radians(34.0784)
    x, y, z = -n * math.sin(lat), e, n * math.cos(lat)
    i, j = torch.triu_indices(27, 27, 1, device=DEV)
    bx, by, bz = x[j] - x[i], y[j] - y[i], z[j] - z[i]
    dumps = -(-rows // BASELINES)
    step = min(10.0, 8 * 3600.0 / dumps)
    start = -2.0e4 + 8.0e3 * r[27]
    H = (start + step * torch.arange(dumps, device=DEV, dtype=F64)) * (2 * math.pi / 86164.0905)
    dec = math.radians(30.0) + math.radians(20.0) * r[28]
    sH, cH, sd, cd = torch.sin(H)[:, None], torch.cos(H)[:, None], torch.sin(dec), torch.cos(dec)
    u = sH * bx + cH * by
    v = -sd * cH * bx + sd * sH * by + cd * bz
    w = cd * cH * bx - cd * sH * by + sd * bz
    return tuple(a.reshape(-1)[:rows].contiguous() for a in (u, v, w))


def _sky_vis(u, v, w, image, cell, g, noise=0.01):
    """Visibilities of eight point sources and noise, complex64."""
    p = torch.rand((8, 3), generator=g, device=DEV, dtype=F64)
    out = torch.zeros(u.numel(), device=DEV, dtype=C64)
    for l, m, f in ((p - 0.5) * image * cell * 0.5 + torch.tensor([0.0, 0.0, 1.0], device=DEV)).tolist():
        n1 = math.sqrt(1.0 - l * l - m * m) - 1.0
        turns = u * l + v * m + w * n1
        ph = (-2.0 * math.pi) * (turns - torch.floor(turns)).to(F32)
        out += torch.polar(torch.full_like(ph, f), ph)
    out += noise * torch.randn(u.numel(), generator=g, device=DEV, dtype=C64)
    return out


def _model(image, g, planes=None):
    """Sparse positive components, as CLEAN leaves them."""
    shape = (image, image) if planes is None else (planes, image, image)
    r = torch.rand(shape, generator=g, device=DEV)
    return torch.where(r > 0.9995, (r - 0.9995) * 2000.0, torch.zeros_like(r))


_CTX, _KEPT = [], {}


def _ctx():
    if not _CTX:
        _CTX.append(cc.Context(0))
        _CTX[0].set_timings(False)
    return _CTX[0]


def _gridder(case, f_hi=1.4e9, oversampling=100):
    """The gridder and W-projector of an image geometry, kept as a program keeps them."""
    planes, smin, smax = (case.get(k, 0) for k in ("planes", "smin", "smax"))
    key = (case["image"], f_hi, oversampling, planes, smin, smax)
    if key not in _KEPT:
        cell = _cell(case["image"], f_hi)
        gg = cc.StandardGridder(_ctx(), cc.ImageGeometry(case["image"], case["image"], cell, cell),
                                oversampling=oversampling)
        gw = None
        if planes:
            # the headline's oversampling of 8 with given supports, the defaults otherwise
            gw = cc.WProjector(gg, 1.0, planes=planes, sampling=8 if smin else None,
                               support_law=(smin, smax) if smin else None)
        _KEPT[key] = gg, gw
    return _KEPT[key]


def _batch(case, seed):
    g = _gen(seed)
    um, vm, wm = _tracks(case["rows"], _radius(case["image"]), g)
    s = 1.4e9 / C_LIGHT
    u, v, w = um * s, vm * s, wm * s
    vis = _sky_vis(u, v, w, case["image"], _cell(case["image"]), g)
    wt = 0.5 + 1.5 * torch.rand(case["rows"], generator=g, device=DEV)
    return g, u, v, w, vis, wt


def _cube_arrays(case, seed):
    g = _gen(seed)
    R, C = case["rows"], case["channels"]
    um, vm, _ = _tracks(R, _radius(case["image"]), g)
    freqs = np.linspace(1.0e9, 2.0e9, C)
    vis = torch.randn((C, R), generator=g, device=DEV, dtype=C64)
    vis += 1.0
    wt = torch.randint(1, 5, (C, R), generator=g, device=DEV, dtype=U8).to(F32) * 0.25
    frac = (255.0 * 0.6 * torch.rand((C, 1), generator=g, device=DEV)).to(U8)
    flags = (torch.randint(0, 256, (C, R), generator=g, device=DEV, dtype=U8) < frac).to(U8)
    return g, um, vm, freqs / C_LIGHT, vis, wt, flags


def _row_arrays(case, seed):
    g = _gen(seed)
    R, C, K = case["rows"], case["channels"], case["corr"]
    uvw = torch.stack(_tracks(R, 5000.0, g), 1).contiguous()
    ls = np.linspace(1.0e9, 2.0e9, C) / C_LIGHT
    data = torch.randn((R, C, K), generator=g, device=DEV, dtype=C64)
    # one sample in ten flagged, in all its correlations, as interference is
    flag = torch.zeros((R * C, K), device=DEV, dtype=U8)
    tens = R * C // 10
    flag[10 * torch.arange(tens, device=DEV) + torch.randint(0, 10, (tens,), generator=g, device=DEV)] = 1
    flag = flag.reshape(R, C, K)
    shape = (R, C, K) if case["spectrum"] else (R, K)
    wt = 0.5 + torch.rand(shape, generator=g, device=DEV)
    return uvw, ls, data, flag, wt


def _hogbom_arrays(case, seed):
    """A PSF from binned tracks and the dirty image of forty sources under it."""
    g = _gen(seed)
    n = case["image"]
    um, vm, _ = _tracks(200000, 1000.0, g)
    s = n / (3.0 * 1.8 * 1000.0)
    cover = torch.zeros((n, n), device=DEV)
    ix, iy = (torch.floor(um * s).long() % n), (torch.floor(vm * s).long() % n)
    cover.index_put_((ix, iy), torch.ones((), device=DEV))
    cover.index_put_(((-ix) % n, (-iy) % n), torch.ones((), device=DEV))
    psf = torch.fft.fftshift(torch.fft.ifft2(cover).real)
    psf = (psf / psf.max()).contiguous()
    sky = torch.zeros((n, n), device=DEV)
    at = (n * (0.25 + 0.5 * torch.rand((40, 2), generator=g, device=DEV))).long()
    flux = 10.0 ** (-2.0 * torch.rand(40, generator=g, device=DEV))
    sky.index_put_((at[:, 0], at[:, 1]), flux, accumulate=True)
    dirty = torch.fft.ifft2(torch.fft.fft2(sky) * torch.fft.fft2(torch.fft.ifftshift(psf))).real
    dirty = (dirty + 1e-3 * torch.randn((n, n), generator=g, device=DEV)).contiguous()
    mask = None
    if case["boxed"]:
        mask = torch.zeros((n, n), device=DEV, dtype=U8)
        mask[n // 5:n - n // 5, n // 5:n - n // 6] = 1
    return psf, dirty, mask


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "rows":
        uvw, ls, data, flag, wt = _row_arrays(case, seed)
        st["runs"] = cc.RowRuns(uvw, ls, data, flag, None if case["spectrum"] else wt,
                                wt if case["spectrum"] else None)
        st["pol"] = cc.Polarization.for_plane("I", [5, 8] if case["corr"] == 2 else [5, 6, 7, 8])
        return st
    if kind == "hogbom":
        st["psf"], st["dirty"], st["mask"] = _hogbom_arrays(case, seed)
        st["model"] = torch.zeros_like(st["dirty"])
        return st
    if kind in ("cube", "cube_refresh"):
        gg, _ = _gridder(case, 2.0e9, 128)
        g, um, vm, ls, vis, wt, flags = _cube_arrays(case, seed)
        st["g"] = gg
        cube = cc.CubeBatch(um, vm, ls, vis, wt, flags)
        if kind == "cube":
            gs = (case["channels"],) + tuple(gg.grid_shape())
            st["cube"] = cube
            st["grids"] = torch.randn(gs, generator=g, device=DEV, dtype=C64)
            st["out"] = (torch.empty(gs, device=DEV, dtype=F32), torch.empty(gs, device=DEV, dtype=C64),
                         torch.empty((case["channels"], case["rows"]), device=DEV, dtype=C64))
        else:
            st["plan"] = cc.CubePlan(gg, cube, "briggs", 0.5)
            st["models"] = _model(case["image"], g, case["channels"])
            st["states"] = st["plan"].dirty_images()[2]
        return st
    gg, gw = _gridder(case)
    g, u, v, w, vis, wt = _batch(case, seed)
    b = cc.VisibilityBatch(u, v, vis, wt, w)
    st.update(g=gg, w=gw, batch=b)
    if kind == "pair":
        st["model"] = _model(case["image"], g).requires_grad_(True)
        st["upstream"] = torch.randn(case["rows"], generator=g, device=DEV, dtype=C64)
    elif kind == "plan":
        st["grid"] = torch.randn(gg.grid_shape(), generator=g, device=DEV, dtype=C64)
    elif kind == "refresh":
        st["model"] = _model(case["image"], g)
        st["state"] = cc.dirty_image(gg, b, gw)[2]
        st["plan"] = cc.Plan(gg, b, gw)
        del st["batch"]
    return st


def _sums(s):
    return {"norm": float(s.normalization_sumwt), "reported": float(s.reported_sumwt),
            "gridded": s.gridded_samples, "skipped": s.skipped_samples,
            "records": s.unique_records, "taps": s.taps}


def run(st):
    kind = st["kind"]
    if kind == "dirty":
        psf, res, state, sums = cc.dirty_image(st["g"], st["batch"], st["w"])
        return {"psf": psf, "residual": res, "peak": float(state.psf_peak), "sums": _sums(sums)}
    if kind == "pair":
        pred = ag.forward(st["model"], st["g"], st["batch"], st["w"])
        grad, = torch.autograd.grad(pred, st["model"], st["upstream"])
        return {"pred": pred.detach(), "grad": grad}
    if kind == "plan":
        p = cc.Plan(st["g"], st["batch"], st["w"])
        psf, dirty = p.grid_dirty()
        return {"psf": psf, "dirty": dirty, "pred": p.degrid(st["grid"]), "sums": _sums(p.sums)}
    if kind == "refresh":
        return {"residual": st["plan"].residual_image(st["model"], st["state"])}
    if kind == "cube":
        psf, dirty, pred, sums = cc.cube_grid_degrid(st["g"], st["cube"], st["grids"], "briggs", 0.5,
                                                     out=st["out"])
        return {"psf": psf, "dirty": dirty, "pred": pred,
                "norm": np.array([s.normalization_sumwt for s in sums]),
                "gridded": np.array([s.gridded_samples for s in sums]),
                "skipped": np.array([s.skipped_samples for s in sums])}
    if kind == "cube_refresh":
        return {"residual": st["plan"].residual_images(st["models"], st["states"])}
    if kind == "hogbom":
        o = cc.run_hogbom_minor_cycle(_ctx(), st["model"], st["dirty"], st["psf"], 0.1,
                                      st["case"]["niter"], mask=st["mask"])
        return {"model": o.model, "residual": o.residual, "at": o.positions, "peaks": o.peaks,
                "fluxes": o.fluxes, "actual": o.actual_updates}
    if kind == "weights":
        wt, f2 = cc.apply_weighting(st["g"], st["batch"], st["case"]["mode"], 0.5)
        return {"weight": wt, "f2": np.float32(f2)}
    b, du, dv = cc.prepare_row_runs(_ctx(), st["runs"], st["pol"])
    return {"u": b.u_lambda, "v": b.v_lambda, "w": b.w_lambda, "weight": b.weight,
            "factor": b.sumwt_factor, "gridable": b.gridable, "vis": b.visibility, "du": du, "dv": dv}


# ---- necessary work --------------------------------------------------------------
def _supports(case):
    p = max(case["planes"], 1)
    if not case["planes"]:
        return [3]
    if not case["smin"]:
        return [5]
    return [case["smin"] + round((case["smax"] - case["smin"]) * k / max(p - 1, 1)) for k in range(p)]


def work(case):
    """Inputs read once and outputs written once; flops of the taps (8 per real kernel
    value and polarisation pair, 12 per complex one) and 2.5 N log2 N per real transform."""
    kind, n = case["kind"], case.get("image", 0)
    R = case["rows"] if kind != "hogbom" else 0
    G = float(1.2 * n) ** 2
    fft = 2.5 * G * math.log2(max(G, 2.0))
    if kind in ("dirty", "pair", "plan", "refresh"):
        s = _supports(case)
        taps = R * sum((2 * k + 1) ** 2 for k in s) / len(s)
        per = 12.0 if case["planes"] else 6.0
        coords = 24 if case["planes"] else 16
        if kind == "dirty":
            return {"bytes": R * (coords + 12) + 8.0 * n * n, "flops": taps * per + 2 * fft}
        if kind == "pair":
            return {"bytes": R * (2 * coords + 16) + 8.0 * n * n, "flops": 1.33 * taps * per + 2 * fft}
        if kind == "plan":
            return {"bytes": R * (coords + 20) + 24.0 * G, "flops": 1.67 * taps * per}
        return {"bytes": R * 20 + 8.0 * n * n, "flops": 1.33 * taps * per + 2 * fft}
    if kind in ("cube", "cube_refresh"):
        C = case["channels"]
        S = float(R) * C
        if kind == "cube":
            return {"bytes": 16.0 * R + S * 21 + C * G * 20, "flops": S * 0.7 * 49 * 10}
        return {"bytes": S * 0.7 * 20 + C * n * n * 8.0, "flops": S * 0.7 * 49 * 8 + 2 * C * fft}
    if kind == "hogbom":
        # the subtraction and the search touch every pixel of every iteration
        return {"bytes": 16.0 * n * n, "flops": 3.0 * n * n * case["niter"]}
    if kind == "weights":
        return {"bytes": R * 24.0, "flops": R * 20.0}
    K = 2 * R * case["channels"]
    wt = 4 * K if case["spectrum"] else 8 * R
    return {"bytes": 24.0 * R + 9.0 * K + wt + 57.0 * R * case["channels"] * 0.9,
            "flops": 12.0 * R * case["channels"]}


# ---- the same in 64 bits ---------------------------------------------------------
def _padded(n):
    p = max(int(math.floor(1.2 * n - 0.5)), n)
    p += p % 2
    while True:
        v = p
        for f in (2, 3, 5):
            while v > 1 and v % f == 0:
                v //= f
        if v == 1:
            return p
        p += 2


def _grdsf(nu):
    """The rational approximation of the zero-order prolate spheroidal function."""
    nu = np.asarray(nu, np.float64)
    p = (np.array([8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1]),
         np.array([4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2]))
    q = (np.array([1.0, 8.212018e-1, 2.078043e-1]), np.array([1.0, 9.599102e-1, 2.918724e-1]))
    out = np.zeros_like(nu)
    for k, (end, m) in enumerate(((0.75, nu < 0.75), (1.0, (nu >= 0.75) & (nu <= 1.0)))):
        d = nu[m] ** 2 - end * end
        out[m] = np.polyval(p[k][::-1], d) / np.polyval(q[k][::-1], d)
    return out


def _axis(n):
    return _grdsf(np.clip(np.abs(np.arange(n) - n / 2.0) / (n / 2.0), 0.0, 1.0))


def _taps(os_):
    half = os_ // 2
    off, t = np.meshgrid(np.arange(-half, half + 1), np.arange(-3, 4), indexing="ij")
    nu = np.abs(t * os_ + off) / (3.0 * os_)
    rows = np.where(nu < 1.0, (1.0 - np.minimum(nu, 1.0) ** 2) * _grdsf(np.minimum(nu, 1.0)), 0.0)
    return torch.as_tensor(rows / rows.sum(1, keepdims=True), device=DEV)


def _nearest(x):
    return torch.sign(x) * torch.floor(torch.abs(x) + 0.5)


class _Exact:
    """The grid geometry of an image and its transforms in 64 bits."""

    def __init__(self, n, cell, oversampling):
        self.n, self.cell, self.os = n, cell, oversampling
        self.G = _padded(n)
        self.blc = (self.G - n + (1 if self.G % 2 == 0 else 0)) // 2
        self.du = 1.0 / (self.G * cell)
        a = _axis(self.G)
        corr = torch.as_tensor(np.where(a > 1e-6, 1.0 / np.where(a > 1e-6, a, 1.0), 0.0), device=DEV)
        self.corr = corr[self.blc:self.blc + n]
        self.taps = _taps(oversampling)
        self.sinc = None

    def plan(self, u, v):
        """Start cells and tap rows; a mask of the samples that grid."""
        out, ok = [], None
        for x in (u / self.du + self.G / 2.0, -v / self.du + self.G / 2.0):
            a = _nearest(x)
            row = _nearest((a - x) * self.os).long() + self.os // 2
            good = (a >= 3) & (a + 3 < self.G) & (row >= 0) & (row < self.taps.shape[0])
            ok = good if ok is None else ok & good
            out += [a.long() - 3, row.clamp(0, self.taps.shape[0] - 1)]
        return out, ok

    def windows(self, u, v):
        """Chunks of (samples, flat cells [m, 49], tap products [m, 49])."""
        (x0, rx, y0, ry), ok = self.plan(u, v)
        at = torch.nonzero(ok).reshape(-1)
        k = torch.arange(7, device=DEV)
        for i in at.split(1 << 19):
            cell = (x0[i][:, None, None] + k[:, None]) * self.G + y0[i][:, None, None] + k
            t = self.taps[rx[i]][:, :, None] * self.taps[ry[i]][:, None, :]
            yield i, cell.reshape(len(i), -1), t.reshape(len(i), -1).to(C128)

    def image(self, grid, scale):
        n, b = self.n, self.blc
        raw = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(grid)))
        f = self.corr[:, None] * self.corr[None, :]
        if self.sinc is not None:
            f = f / (self.sinc[:, None] * self.sinc[None, :])
        return raw[b:b + n, b:b + n].real * f * scale

    def model_grid(self, model):
        n, b = self.n, self.blc
        full = torch.zeros((self.G, self.G), device=DEV, dtype=C128)
        f = self.corr[:, None] * self.corr[None, :]
        if self.sinc is not None:
            f = f * self.sinc[:, None] * self.sinc[None, :]
        full[b:b + n, b:b + n] = (model.to(F64) * f).to(C128)
        return torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(full)))

    def grid(self, windows, values):
        """Sums of each listed value times its window's taps, one grid per value."""
        out = [torch.zeros(2 * self.G * self.G, device=DEV, dtype=F64) for _ in values]
        for i, cell, t in windows:
            for o, val in zip(out, values):
                add = torch.view_as_real(val[i][:, None] * t).reshape(-1)
                o.index_add_(0, (2 * cell[:, :, None] + torch.arange(2, device=DEV)).reshape(-1), add)
        return [torch.view_as_complex(o.reshape(self.G, self.G, 2)) for o in out]

    def degrid(self, windows, grid, n):
        out = torch.zeros(n, device=DEV, dtype=C128)
        flat = grid.reshape(-1)
        for i, cell, t in windows:
            out[i] = (flat[cell] * t.conj()).sum(1)
        return out


class _ExactW(_Exact):
    """W-projection: the kernels of every plane and their windows."""

    def __init__(self, n, cell, planes, smin, smax):
        super().__init__(n, cell, 100)
        self.planes = planes
        s = self.s = 8 if smin else 4
        G, r = self.G, (s + 1) // 2
        inner, quarter = max(G // s, 2), G // 2 - 1
        half = inner // 2
        self.w_scale = (planes - 1) ** 2 / (0.25 / cell)
        c = torch.as_tensor(_axis(inner), device=DEV)
        ix = torch.arange(inner, device=DEV) - half
        l = cell * s * ix.to(F64)
        rsq = l[:, None] ** 2 + l[None, :] ** 2
        self.kernels, self.support, peak = [], [], None
        for p in range(planes):
            ph = 2.0 * math.pi * (p * p / self.w_scale) * (torch.sqrt(1.0 - rsq) - 1.0)
            buf = torch.zeros((G, G), device=DEV, dtype=C128)
            at = ix % G
            buf[at[:, None], at[None, :]] = torch.polar(c[:, None] * c[None, :], ph)
            T = torch.fft.fft2(buf)
            if peak is None:
                peak = float(T[0, 0].abs())
            T = T / peak
            if smin:
                S = _law(smin, smax, p, planes)
            else:
                a = torch.maximum(T[:quarter, 0].abs(), T[0, :quarter].abs())
                most = max(quarter // s - 1, 1)
                hit = torch.nonzero(a[1:] > 1e-3).reshape(-1)
                S = most if not len(hit) else min(int(math.floor(float(hit[-1] + 1) / s + 0.5)) + 1, most)
            width = S * s + r + 1 if smin else max(min(S * s + r + 1, quarter), 1)
            self.support.append(S)
            self.kernels.append(T[:width, :width].clone())
        S0 = self.support[0]
        k = (torch.arange(-S0, S0 + 1, device=DEV) * s).abs()
        total = float(self.kernels[0][k[:, None], k[None, :]].real.sum())
        self.kernels = [K / total for K in self.kernels]
        x = torch.arange(G, device=DEV, dtype=F64) - G // 2
        sinc = torch.special.sinc(x / (G * s))
        self.sinc = sinc[self.blc:self.blc + n]

    def locate(self, u, v, w):
        loc, off = [], []
        for x in (u / self.du + self.G / 2.0, -v / self.du + self.G / 2.0):
            a = _nearest(x)
            loc.append(a.long())
            off.append(_nearest((a - x) * self.s).long())
        plane = _nearest(torch.sqrt(self.w_scale * w.abs())).clamp(0, self.planes - 1).long()
        S = torch.tensor(self.support, device=DEV)[plane]
        ok = (loc[0] >= S) & (loc[1] >= S) & (loc[0] + S < self.G) & (loc[1] + S < self.G)
        return loc, off, plane, ok

    def windows_w(self, u, v, w):
        loc, off, plane, ok = self.locate(u, v, w)
        for p in range(self.planes):
            S, K = self.support[p], self.kernels[p]
            k = torch.arange(-S, S + 1, device=DEV)
            for i in torch.nonzero(ok & (plane == p)).reshape(-1).split(max((1 << 24) // (2 * S + 1) ** 2, 1)):
                if not len(i):
                    continue
                kx = (k * self.s + off[0][i][:, None]).abs()
                ky = (k * self.s + off[1][i][:, None]).abs()
                t = K[kx[:, :, None], ky[:, None, :]]
                t = torch.where((w[i] > 0)[:, None, None], t.conj(), t)
                cell = (loc[0][i][:, None, None] + k[:, None]) * self.G + loc[1][i][:, None, None] + k
                yield i, cell.reshape(len(i), -1), t.reshape(len(i), -1)


def _law(smin, smax, p, planes):
    return smin + int(math.floor((smax - smin) * p / max(planes - 1, 1) + 0.5))


def _exact_sums(norm, reported, gridded, rows):
    return {"norm": torch.tensor(norm, dtype=F64), "reported": torch.tensor(reported, dtype=F64),
            "gridded": None, "skipped": None, "records": None, "taps": None}


def _exact_single(case, seed):
    kind = case["kind"]
    S = 7 if not case["smin"] else case["smax"]
    if case["rows"] * (2.0 * (S if case["planes"] else 3) + 1.0) ** 2 > MAX_EXACT_TAPS:
        return None
    if case["planes"] and case["planes"] * float(_padded(case["image"])) ** 2 > 4.0e8:
        return None
    g, u, v, w, vis, wt = _batch(case, seed)
    n, R, cell = case["image"], case["rows"], _cell(case["image"])
    if case["planes"]:
        e = _ExactW(n, cell, case["planes"], case["smin"], case["smax"])
        wins = lambda: e.windows_w(u, v, w)  # noqa: E731
        ok, k = e.locate(u, v, w)[3], 2.0
    else:
        e = _Exact(n, cell, 100)
        wins = lambda: e.windows(u, v)  # noqa: E731
        ok, k = e.plan(u, v)[1], 1.0
    wt64, vis128 = wt.to(F64), vis.to(C128)
    if kind == "pair":
        model = _model(n, g)
        up = torch.randn(R, generator=g, device=DEV, dtype=C64).to(C128)
        grad = e.image(e.grid(wins(), [up])[0], 1.0)
        if e.sinc is not None:   # the adjoint multiplies by the sinc the image divides by
            grad = grad * (e.sinc[:, None] * e.sinc[None, :]) ** 2
        return {"pred": e.degrid(wins(), e.model_grid(model), R), "grad": grad * float(e.G) ** 2}
    if kind == "plan":
        grid = torch.randn((e.G, e.G), generator=g, device=DEV, dtype=C64).to(C128)
    norm = reported = float((wt64 * ok).sum())
    if case["planes"]:
        norm = sum(2.0 * float((wt64[i] * t.real.sum(1)).sum()) for i, _, t in wins())
    psf, dirty = e.grid(wins(), [wt64.to(C128), wt64 * vis128])
    if kind == "plan":
        return {"psf": psf, "dirty": dirty, "pred": e.degrid(wins(), grid, R),
                "sums": _exact_sums(norm, reported, int(ok.sum()), R)}
    p = e.image(psf, k / norm)
    peak = float(p.abs().max())
    if kind == "refresh":
        pred = e.degrid(wins(), e.model_grid(_model(n, g)), R)
        return {"residual": e.image(e.grid(wins(), [wt64 * (vis128 - pred)])[0], k / norm / peak)}
    return {"psf": p / peak, "residual": e.image(dirty, k / norm / peak),
            "peak": torch.tensor(peak, dtype=F64), "sums": _exact_sums(norm, reported, 0, R)}


def _density_cells(u, v, n, cell):
    """Rounded cells of (u, v) on the image-sized density grid, and which are inside."""
    x, y = _nearest(u * (n * cell) + n / 2.0), _nearest(-v * (n * cell) + n / 2.0)
    ok = (x >= 1) & (y >= 1) & (x < n) & (y < n)
    return torch.where(ok, x * n + y, torch.zeros_like(x)).long(), ok


def _briggs(density, w, d, ok, mode, robust):
    if mode == "uniform":
        return torch.where(ok & (d > 0), w / torch.where(d > 0, d, torch.ones_like(d)), torch.zeros_like(w)), 0.0
    f2 = (5.0 * 10.0 ** -robust) ** 2 / (float((density * density).sum()) / float(density.sum()))
    return torch.where(ok & (d > 0), w / (d * f2 + 1.0), torch.zeros_like(w)), f2


def _exact_weights(case, seed):
    _, u, v, _, _, wt = _batch(case, seed)
    if case["mode"] == "natural":
        return {"weight": wt.to(F64), "f2": torch.tensor(0.0, dtype=F64)}
    n = case["image"]
    w = wt.to(F64)
    scale = torch.tensor(n * _cell(n), dtype=F32, device=DEV)
    half = torch.tensor(n / 2.0, dtype=F32, device=DEV)
    density = torch.zeros(n * n, device=DEV, dtype=F64)
    # the cell is the truncation of a float32 coordinate by definition
    own = None
    for s in (1.0, -1.0):
        x = -(s * u).to(F32) * scale + half
        y = (s * v).to(F32) * scale + half
        ok = (x >= 1) & (y >= 1) & (x < n) & (y < n)
        c = torch.where(ok, x.long() * n + y.long(), torch.zeros_like(x, dtype=torch.long))
        density.index_add_(0, c, w * ok)
        own = own or (c, ok)
    out, f2 = _briggs(density, w, density[own[0]], own[1], case["mode"], 0.5)
    return {"weight": out, "f2": torch.tensor(f2, dtype=F64)}


def _exact_cube(case, seed):
    R, C, n = case["rows"], case["channels"], case["image"]
    if R * C * 49.0 > MAX_EXACT_TAPS:
        return None
    cell = _cell(n, 2.0e9)
    e = _Exact(n, cell, 128)
    g, um, vm, ls, vis, wt, flags = _cube_arrays(case, seed)
    res = {k: [] for k in ("psf", "dirty", "pred", "norm", "residual")}
    if case["kind"] == "cube":
        grids = torch.randn((C, e.G, e.G), generator=g, device=DEV, dtype=C64)
    else:
        models = _model(n, g, C)
    for c in range(C):
        live = torch.nonzero(flags[c] == 0).reshape(-1)
        u, v = um[live] * float(ls[c]), vm[live] * float(ls[c])
        w, vs = wt[c][live].to(F64), vis[c][live].to(C128)
        density = torch.zeros(n * n, device=DEV, dtype=F64)
        for s in (1.0, -1.0):
            at, ok = _density_cells(s * u, s * v, n, cell)
            density.index_add_(0, at, w * ok)
        at, ok = _density_cells(u, v, n, cell)
        w, _ = _briggs(density, w, density[at], ok, "briggs", 0.5)
        norm = float((w * e.plan(u, v)[1]).sum())
        if case["kind"] == "cube":
            psf, dirty = e.grid(e.windows(u, v), [w.to(C128), w * vs])
            pred = torch.zeros(R, device=DEV, dtype=C128)
            pred[live] = torch.where(w > 0, e.degrid(e.windows(u, v), grids[c].to(C128), len(live)),
                                     torch.zeros_like(vs))
            res["psf"].append(psf.real), res["dirty"].append(dirty), res["pred"].append(pred)
            res["norm"].append(norm)
        else:
            peak = float(e.image(e.grid(e.windows(u, v), [w.to(C128)])[0], 1.0 / norm).abs().max())
            pred = e.degrid(e.windows(u, v), e.model_grid(models[c]), len(live))
            grid, = e.grid(e.windows(u, v), [w * (vs - pred)])
            res["residual"].append(e.image(grid, 1.0 / norm / peak))
    if case["kind"] == "cube_refresh":
        return {"residual": torch.stack(res["residual"])}
    return {"psf": torch.stack(res["psf"]), "dirty": torch.stack(res["dirty"]),
            "pred": torch.stack(res["pred"]), "norm": np.array(res["norm"]),
            "gridded": None, "skipped": None}


def _exact_rows(case, seed):
    uvw, ls, data, flag, wt = _row_arrays(case, seed)
    a, b = 0, case["corr"] - 1
    keep = (flag[:, :, a] == 0) & (flag[:, :, b] == 0)
    r, c = torch.nonzero(keep, as_tuple=True)
    if not case["spectrum"]:
        wt = wt[:, None, :].expand(-1, case["channels"], -1)
    s = torch.as_tensor(ls, device=DEV)[c]
    s32 = s.to(F32).to(F64)
    out = {k: uvw[r, i] * s for i, k in enumerate("uvw")}
    out["weight"] = 0.5 * (wt[:, :, a].to(F64) + wt[:, :, b].to(F64))[keep]
    out["factor"] = torch.full_like(s, 2.0)
    out["gridable"] = None
    out["vis"] = 0.5 * (data[:, :, a].to(C128) + data[:, :, b].to(C128))[keep]
    out["du"], out["dv"] = ((uvw[r, i] * s32).to(F32).to(F64) for i in (0, 1))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "hogbom":
        return None   # a sequence of decisions on float32 values: no 64-bit counterpart
    if kind == "rows":
        return _exact_rows(case, seed)
    if kind == "weights":
        return _exact_weights(case, seed)
    if kind in ("cube", "cube_refresh"):
        return _exact_cube(case, seed)
    return _exact_single(case, seed)
