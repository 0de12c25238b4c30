"""Performance cases of the w-gridder: what users of this library have it do.

Every case goes through the package's public entry points: the ducc0-style
operators of a ``Context``, WSClean's stateful ``WGriddingGridder``, ``Plan``
(facets times output channels), ``Stream`` (chunks from host memory) and
``ImageWeights``.  Observations are Earth-rotation tracks of random arrays
with w rescaled to a stated fraction of the longest baseline; visibilities are
a few point sources plus noise; model images are sparse CLEAN components.

Fields of a case: ``kind`` (see ``run``), the array (``nant`` antennas within
``radius`` metres, log-radial or uniform), ``ntimes`` samples ``cadence``
seconds apart, ``nchan`` channels from ``f0`` to ``f1`` Hz, |w| up to
``wfrac`` of max |uv|, an ``nx`` x ``ny`` image of ``pix`` arcsec pixels,
``eps``, ``precision``, and the options ``weighted``, ``masked`` and ``shift``
(phase centre offset in pixels).
"""
import math

import numpy as np
import torch

from wsclean_b200 import gridder as G

C_LIGHT = 299792458.0
ARCSEC = math.pi / (180 * 3600)
LATITUDE = math.radians(-26.7)

# WSClean's call pattern (v negated, no division by n, sigma up to 2)
WSCLEAN = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)

_BASE = dict(nant=64, radius=3000.0, log_radial=False, ntimes=60, cadence=10.0, nchan=1,
             f0=150e6, f1=150e6, wfrac=0.2, nx=1024, ny=1024, pix=10.0, eps=1e-5,
             precision="mixed", weighted=False, masked=False, shift=0, nsrc=20)


def _case(name, kind, **kw):
    return dict(_BASE, name=name, kind=kind, **kw)


def listed():
    return [
        # a snapshot of a small array imaged for a quick look or by a
        # calibration loop that calls thousands of times: latency and launches
        _case("grid_snapshot", "grid", nant=27, radius=1500.0, ntimes=6, nchan=4, f0=150e6,
              f1=151.5e6, nx=256, ny=256, pix=24.0, eps=1e-4),
        _case("predict_snapshot", "predict", nant=27, radius=1500.0, ntimes=6, nchan=4, f0=150e6,
              f1=151.5e6, nx=256, ny=256, pix=24.0, eps=1e-4),
        # a facet of odd shape, off the phase centre, with weights and flags,
        # as facet imaging and self-calibration grid it
        _case("grid_ragged_facet", "grid", nant=45, radius=4000.0, ntimes=33, nchan=5, f0=143e6,
              f1=147.1e6, nx=742, ny=458, pix=7.3, eps=1e-4, weighted=True, masked=True,
              shift=517, wfrac=0.3),
        # one hour of a 64-station array in double precision to full accuracy
        # (scientific reference images, WSClean's NumT=double)
        _case("grid_fp64", "grid", ntimes=360, nchan=4, f0=150e6, f1=151.5e6, eps=1e-12,
              precision="fp64"),
        _case("predict_fp64", "predict", ntimes=360, nchan=4, f0=150e6, f1=151.5e6, eps=1e-12,
              precision="fp64"),
        # the headline wide field: 8.1M visibilities onto 4096^2, both ways
        _case("grid_field", "grid", nant=128, radius=6000.0, ntimes=997, cadence=8.0, wfrac=0.3,
              nx=4096, ny=4096, pix=5.0, nsrc=50),
        _case("predict_field", "predict", nant=128, radius=6000.0, ntimes=997, cadence=8.0,
              wfrac=0.3, nx=4096, ny=4096, pix=5.0, nsrc=200),
        # the gradient of a weighted chi^2 with respect to the model image:
        # prediction, residual, gridding (gradient-based imaging)
        _case("chi2_gradient", "gradient", nant=128, radius=6000.0, ntimes=400, cadence=8.0,
              wfrac=0.3, nx=2048, ny=2048, pix=8.0, weighted=True, nsrc=200),
        # WSClean's gridder object fed host chunks of a measurement set, in
        # double precision at 1e-5 (its factory's choice at that accuracy);
        # padded image of odd proportions, trimmed result
        _case("dropin_chunks", "dropin", nant=62, radius=3500.0, ntimes=120, nchan=3, f0=140e6,
              f1=144e6, nx=1500, ny=1320, pix=8.0, eps=1e-5, precision="fp64", shift=40),
        # a major cycle (predict, subtract, invert) over facets times output
        # channels, one plan kept for all cycles
        _case("facet_cycle", "facets", nant=96, radius=6000.0, ntimes=60, nchan=16, f0=120e6,
              f1=180e6, nx=3072, ny=3072, pix=10.0, nfacet=3, nout=4, nsrc=40),
        # an observation streamed in chunks from page-locked host memory into
        # a resident 8192^2 grid, predicted and gridded
        _case("stream_wide", "stream", nant=256, radius=20000.0, log_radial=True, ntimes=48,
              cadence=160.0, nchan=16, f0=140e6, f1=190e6, wfrac=0.1, nx=8192, ny=8192, pix=2.0,
              nchunk=4, nsrc=50),
        # Briggs imaging weights of a full observation: grid, finish, look up
        _case("briggs_weights", "weights", nant=128, radius=6000.0, ntimes=500, cadence=8.0,
              nchan=2, f0=148e6, f1=152e6, nx=4096, ny=4096, pix=5.0, weighted=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: any of the kinds above over its range of sizes."""
    kind = rng.choice(["grid", "predict", "grid", "predict", "gradient", "dropin", "facets",
                       "stream", "weights"])
    c = dict(_BASE, kind=kind)
    c["nchan"] = rng.choice([1, 2, 3, 4, 7, 16])
    c["f0"] = rng.uniform(120e6, 160e6)
    c["f1"] = c["f0"] * (1 + 0.004 * (c["nchan"] - 1))
    c["cadence"] = rng.choice([4.0, 8.0, 10.0])
    c["wfrac"] = rng.uniform(0.05, 0.35)
    c["radius"] = rng.uniform(1500.0, 6000.0)
    c["nant"] = rng.randint(24, 128)
    fp64 = rng.random() < 0.35
    c["precision"] = "fp64" if fp64 else "mixed"
    c["eps"] = rng.choice([1e-5, 1e-7, 1e-9, 1e-12]) if fp64 else rng.choice([1e-3, 1e-4, 1e-5])
    lo, hi = 192, (2048 if fp64 else 4096)
    if kind in ("stream", "facets"):
        lo, hi = 1024, 3072
    c["nx"] = 2 * int(_log(rng, lo, hi) / 2)
    c["ny"] = 2 * int(min(max(c["nx"] * rng.uniform(0.5, 1.5), lo), hi) / 2)
    # pixels 2.5 to 5 to the resolution of the longest baseline, in a field of
    # at most 7 degrees
    lam = C_LIGHT / c["f1"]
    pix = lam / (2 * c["radius"]) / rng.uniform(2.5, 5.0) / ARCSEC
    c["pix"] = min(pix, 25000.0 / max(c["nx"], c["ny"]))
    bl = c["nant"] * (c["nant"] - 1) // 2
    most = 4e6 if kind in ("facets", "gradient") else (3e6 if fp64 else 8e6)
    c["ntimes"] = max(2, int(_log(rng, 8e3, most) / bl / c["nchan"]))
    c["weighted"] = rng.random() < 0.5
    c["masked"] = kind in ("grid", "predict") and rng.random() < 0.3
    c["shift"] = rng.choice([0, 0, rng.randint(1, 300)])
    c["nsrc"] = rng.randint(10, 100)
    if kind == "dropin":
        c.update(weighted=False, precision="fp64" if c["eps"] <= 1.01e-5 else "mixed")
    if kind == "facets":
        c.update(precision="mixed", eps=rng.choice([1e-4, 1e-5]), nchan=8, shift=0,
                 f1=c["f0"] * 1.2, nfacet=rng.choice([2, 3]), nout=rng.choice([2, 4]))
        c["ntimes"] = max(2, c["ntimes"] * c["nchan"] // 64)
    if kind == "stream":
        c.update(precision="mixed", eps=rng.choice([1e-4, 1e-5]), weighted=False,
                 nchunk=rng.randint(2, 5))
    if kind == "weights":
        c.update(weighted=True, shift=0)
    return c


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _uvw(c, rng, dev):
    """uvw in metres, rows time-major, on the device."""
    n = c["nant"]
    if c["log_radial"]:
        r = 50.0 * (c["radius"] / 50.0) ** rng.uniform(0, 1, n)
    else:
        r = c["radius"] * np.sqrt(rng.uniform(0, 1, n))
    r[0], r[1] = c["radius"], c["radius"]   # the array's stated extent
    phi = rng.uniform(0, 2 * np.pi, n)
    phi[1] = phi[0] + np.pi
    e, nn = r * np.cos(phi), r * np.sin(phi)
    xyz = np.stack([-math.sin(LATITUDE) * nn, e, math.cos(LATITUDE) * nn], axis=1)
    i, j = np.triu_indices(n, k=1)
    b = torch.as_tensor(xyz[j] - xyz[i], device=dev)
    nt = c["ntimes"]
    span = nt * c["cadence"] / 3600.0 * (2 * math.pi / 24.0)
    H = torch.linspace(-0.5, 0.5, nt, dtype=torch.float64, device=dev)[:, None] * span
    sH, cH = torch.sin(H), torch.cos(H)
    dec = math.radians(-30.0)
    sd, cd = math.sin(dec), math.cos(dec)
    bx, by, bz = b[:, 0], b[:, 1], b[:, 2]
    u = sH * bx + cH * by
    v = -sd * cH * bx + sd * sH * by + cd * bz
    w = cd * cH * bx - cd * sH * by + sd * bz
    uvw = torch.stack([u.reshape(-1), v.reshape(-1), w.reshape(-1)], dim=1)
    uvmax = torch.hypot(uvw[:, 0], uvw[:, 1]).max()
    uvw[:, 2] *= c["wfrac"] * uvmax / uvw[:, 2].abs().max()
    return uvw.contiguous()


def _freq(c):
    return np.linspace(c["f0"], c["f1"], c["nchan"])


def _centre(c):
    return c["shift"] * c["pix"] * ARCSEC, -0.6 * c["shift"] * c["pix"] * ARCSEC


def _sources(rng, n, nx, ny):
    """Components away from the edges: pixel indices and fluxes (power law)."""
    ix = rng.choice(np.arange(int(0.1 * nx), int(0.9 * nx)), n)
    iy = rng.choice(np.arange(int(0.1 * ny), int(0.9 * ny)), n)
    a = -0.6
    flux = (0.01 ** a + rng.uniform(0, 1, n) * (10.0 ** a - 0.01 ** a)) ** (1.0 / a)
    return ix, iy, flux


def _lmn(c, ix, iy, nx, ny, cx, cy, dev):
    """(l, m with v's sign folded in, -(n - 1)) of pixels, 3 x count."""
    p = c["pix"] * ARCSEC
    ix = torch.as_tensor(ix, dtype=torch.float64, device=dev)
    iy = torch.as_tensor(iy, dtype=torch.float64, device=dev)
    lx = cx + (ix - nx / 2) * p
    my = -cy + (iy - ny / 2) * p
    r2 = lx * lx + my * my
    nm1 = -r2 / (torch.sqrt(1 - r2) + 1)
    return torch.stack([lx, -my, -nm1])


def _dft_vis(uvw, freq, lmn, flux):
    """sum_s flux_s exp(-2 pi i (u l + v m + w (n-1))), rows x channels, 64 bits."""
    flux = torch.as_tensor(flux, dtype=torch.float64, device=uvw.device)
    out = torch.empty((uvw.shape[0], len(freq)), dtype=torch.complex128, device=uvw.device)
    step = max(1, (1 << 26) // max(1, flux.numel()))
    for k, f in enumerate(freq):
        for r in range(0, uvw.shape[0], step):
            t = (uvw[r:r + step] * (f / C_LIGHT)) @ lmn
            t = (t - torch.round(t)) * (2 * math.pi)
            out[r:r + step, k] = torch.complex(torch.cos(t) @ flux, -(torch.sin(t) @ flux))
    return out


def _dft_image(c, uvw, freq, vis, nx, ny, cx, cy):
    """Re sum_k vis_k exp(+2 pi i ...) at every pixel, 64 bits."""
    dev = uvw.device
    f = torch.as_tensor(freq / C_LIGHT, dtype=torch.float64, device=dev)
    b = (uvw[:, None, :] * f[None, :, None]).reshape(-1, 3).contiguous()
    v = vis.reshape(-1)
    vr, vi = v.real.double().contiguous(), v.imag.double().contiguous()
    out = torch.empty(nx * ny, dtype=torch.float64, device=dev)
    step = max(1, (1 << 28) // b.shape[0])
    for p in range(0, nx * ny, step):
        at = torch.arange(p, min(p + step, nx * ny), device=dev)
        lmn = _lmn(c, at // ny, at % ny, nx, ny, cx, cy, dev)
        t = lmn.T @ b.T
        t -= torch.round(t)
        t *= 2 * math.pi
        out[p:p + step] = torch.cos(t) @ vr - torch.sin(t) @ vi
    return out.reshape(nx, ny)


def _noise(shape, gen, dtype, sigma):
    dev = gen.device
    re = torch.randn(shape, generator=gen, device=dev, dtype=dtype) * sigma
    im = torch.randn(shape, generator=gen, device=dev, dtype=dtype) * sigma
    return torch.complex(re, im)


def _vis(c, uvw, freq, rng, gen, n=8):
    """A few bright sources plus noise, in the precision of the case."""
    cx, cy = _centre(c)
    ix, iy, flux = _sources(rng, n, c["nx"], c["ny"])
    v = _dft_vis(uvw, freq, _lmn(c, ix, iy, c["nx"], c["ny"], cx, cy, uvw.device), flux)
    real = torch.float64 if c["precision"] == "fp64" and c["kind"] != "dropin" else torch.float32
    v = v.to(torch.complex128 if real == torch.float64 else torch.complex64)
    return v + _noise(v.shape, gen, real, 0.1)


def _facets(c):
    """Uneven facets of the field: sizes and phase centres."""
    n, p = c["nfacet"], c["pix"] * ARCSEC
    cuts = [0.0] + [(k + 1 + 0.25 * (-1) ** k) / n for k in range(n - 1)] + [1.0]
    xs = [2 * int(round(q * c["nx"] / 2)) for q in cuts]
    ys = [2 * int(round(q * c["ny"] / 2)) for q in cuts]
    out = []
    for a in range(n):
        for b in range(n):
            nx, ny = xs[a + 1] - xs[a], ys[b + 1] - ys[b]
            dx = 0.5 * (xs[a] + xs[a + 1]) - c["nx"] / 2
            dy = 0.5 * (ys[b] + ys[b + 1]) - c["ny"] / 2
            # (negated v: the image's m axis runs opposite to center_y)
            out.append(dict(npix_x=nx, npix_y=ny, center_x=dx * p, center_y=-dy * p))
    return out


def _jobs(c):
    per = c["nchan"] // c["nout"]
    return [dict(f, chan_begin=k * per, chan_end=(k + 1) * per)
            for k in range(c["nout"]) for f in _facets(c)]


def _inputs(c, seed):
    """Everything that is drawn from the seed, as a dict."""
    dev = _device()
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    s = dict(uvw=_uvw(c, rng, dev), freq=_freq(c), wgt=None, mask=None)
    kind = c["kind"]
    shape = (s["uvw"].shape[0], c["nchan"])
    if c["weighted"]:
        s["wgt"] = torch.rand(shape, generator=gen, device=dev, dtype=torch.float32) * 1.5 + 0.5
    if c["masked"]:
        s["mask"] = (torch.rand(shape, generator=gen, device=dev) > 0.07).to(torch.uint8)
    if kind in ("grid", "gradient", "facets", "stream", "dropin"):
        s["vis"] = _vis(c, s["uvw"], s["freq"], rng, gen)
    if kind in ("predict", "gradient", "stream"):
        s["src"] = _sources(rng, c["nsrc"], c["nx"], c["ny"])
        s["img"] = _model(c, s["src"], c["nx"], c["ny"], dev)
    if kind == "facets":
        s["srcs"] = [_sources(rng, c["nsrc"], j["npix_x"], j["npix_y"]) for j in _jobs(c)]
        s["imgs"] = [_model(c, q, j["npix_x"], j["npix_y"], dev)
                     for q, j in zip(s["srcs"], _jobs(c))]
    return s


def _model(c, src, nx, ny, dev):
    img = np.zeros((nx, ny))
    np.add.at(img, (src[0], src[1]), src[2])
    real = torch.float64 if c["precision"] == "fp64" else torch.float32
    return torch.as_tensor(img, device=dev).to(real)


def _args(c):
    cx, cy = _centre(c)
    return dict(WSCLEAN, center_x=cx, center_y=cy, precision=c["precision"])


def prepare(case, seed):
    c = case
    s = _inputs(c, seed)
    kind, p = c["kind"], c["pix"] * ARCSEC
    s.update(case=c, px=p)
    s.pop("src", None)
    s.pop("srcs", None)
    if kind in ("grid", "predict", "gradient"):
        s["ctx"] = G.Context()
    elif kind == "dropin":
        # the measurement set's columns, in host memory, in two chunks
        n = s["uvw"].shape[0]
        uvw, vis = s["uvw"].cpu().numpy(), s.pop("vis").cpu().numpy()
        cuts = [0, n // 2 + 1, n]
        s["chunks"] = [(uvw[a:b].copy(), vis[a:b].copy()) for a, b in zip(cuts, cuts[1:])]
        cx, cy = _centre(c)
        tx, ty = 2 * int(0.45 * c["nx"]), 2 * int(0.45 * c["ny"])
        s["gridder"] = G.WGriddingGridder(c["nx"], c["ny"], tx, ty, p, p, -cx, -cy,
                                          epsilon=c["eps"], precision=c["precision"])
    elif kind == "facets":
        s["plan"] = G.Plan(s["uvw"], s["freq"], p, p, c["eps"], jobs=_jobs(c), wgt=s["wgt"],
                           negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0,
                           precision=c["precision"])
        del s["uvw"]
    elif kind == "stream":
        uvw, vis = s.pop("uvw").cpu(), s.pop("vis").cpu()
        ext = G.data_extent(uvw.numpy(), s["freq"])
        n = uvw.shape[0]
        cuts = [n * k // c["nchunk"] for k in range(c["nchunk"] + 1)]
        s["chunks"] = [(uvw[a:b].contiguous().pin_memory(), vis[a:b].contiguous().pin_memory(),
                        torch.empty((b - a, c["nchan"]), dtype=torch.complex64).pin_memory())
                       for a, b in zip(cuts, cuts[1:])]
        s["image"] = torch.zeros((c["nx"], c["ny"]), dtype=torch.float32, device=s["img"].device)
        s["ctx"] = G.Context()
        s["stream"] = G.Stream(s["freq"], c["nx"], c["ny"], p, p, c["eps"], ext,
                               nvis=n * c["nchan"], context=s["ctx"], **_args(c))
    elif kind == "weights":
        s["ctx"] = G.Context()
    return s


def run(state):
    s, c = state, state["case"]
    kind, px = c["kind"], state["px"]
    if kind == "grid":
        return s["ctx"].ms2dirty(s["uvw"], s["freq"], s["vis"], c["nx"], c["ny"], px, px, c["eps"],
                                 wgt=s["wgt"], mask=s["mask"], **_args(c))
    if kind == "predict":
        dt = np.complex128 if c["precision"] == "fp64" else np.complex64
        return s["ctx"].dirty2ms(s["uvw"], s["freq"], s["img"], px, px, c["eps"], wgt=s["wgt"],
                                 mask=s["mask"], vis_dtype=dt, **_args(c))
    if kind == "gradient":
        # d/dI sum_k w_k |V_k - (A I)_k|^2 = -2 A^T w (V - A I)
        dt = np.complex128 if c["precision"] == "fp64" else np.complex64
        model = s["ctx"].dirty2ms(s["uvw"], s["freq"], s["img"], px, px, c["eps"], vis_dtype=dt,
                                  **_args(c))
        res = s["vis"] - model
        g = s["ctx"].ms2dirty(s["uvw"], s["freq"], res, c["nx"], c["ny"], px, px, c["eps"],
                              wgt=s["wgt"], **_args(c))
        return {"gradient": g.mul_(-2.0), "model": model}
    if kind == "dropin":
        g = s["gridder"]
        g.InitializeInversion()
        for uvw, vis in s["chunks"]:
            g.AddInversionData(uvw, s["freq"], vis)
        g.FinalizeImage(1.0 / sum(v.size for _, v in s["chunks"]))
        return g.RealImage()
    if kind == "facets":
        model = s["plan"].dirty2ms(s["imgs"])
        images = s["plan"].ms2dirty(s["vis"] - model)
        return {"model": model, "images": images}
    if kind == "stream":
        st = s["stream"]
        st.predict_begin(s["img"])
        for uvw, _, out in s["chunks"]:
            st.predict(uvw, vis=out)
        for uvw, vis, _ in s["chunks"]:
            st.add(uvw, vis)
        st.finish(dirty=s["image"])
        return {"model": [o for _, _, o in s["chunks"]], "image": s["image"]}
    if kind == "weights":
        with G.ImageWeights("briggs", 0.0, c["nx"], c["ny"], px, px, context=s["ctx"]) as w:
            w.grid(s["uvw"], s["freq"], s["wgt"])
            w.finish()
            return w.apply(s["uvw"], s["freq"], s["wgt"])
    raise ValueError(kind)


# ---------------------------------------------------------- work and truth


def _counts(c):
    rows = c["nant"] * (c["nant"] - 1) // 2 * c["ntimes"]
    return rows, rows * c["nchan"]


def work(case):
    """Inputs once, outputs once; multiply-adds of the kernel footprints and
    one transform of an oversampled plane (the w planes come on top)."""
    c = case
    rows, nvis = _counts(c)
    wide = c["precision"] == "fp64"
    cs = 16 if wide and c["kind"] != "dropin" else 8
    npix, ps = c["nx"] * c["ny"], 8 if wide else 4
    W = math.ceil(-math.log10(c["eps"])) + 2
    n = 1.5 * c["nx"] * 1.5 * c["ny"]
    one = 4.0 * nvis * W ** 3 + 5.0 * n * math.log2(n)
    data = rows * 24 + nvis * cs + npix * ps
    if c["weighted"]:
        data += nvis * 4
    if c["masked"]:
        data += nvis
    kind = c["kind"]
    if kind == "weights":
        return {"bytes": 2 * rows * 24 + nvis * 12 + npix * 8, "flops": 20.0 * nvis}
    if kind == "dropin":
        return {"bytes": rows * 24 + nvis * 8 + npix * 4, "flops": one}
    if kind == "gradient":
        return {"bytes": 2 * data + nvis * 3 * cs, "flops": 2 * one}
    if kind == "facets":
        return {"bytes": 2 * data + nvis * 3 * cs, "flops": 2 * one * c["nfacet"] ** 2}
    if kind == "stream":
        return {"bytes": 2 * data, "flops": 2 * one}
    return {"bytes": data, "flops": one}


def exact(case, seed):
    """The direct Fourier transform in 64 bits, where it is affordable."""
    c = case
    _, nvis = _counts(c)
    kind = c["kind"]
    npix = c["nx"] * c["ny"]
    if kind == "weights":
        return _exact_weights(c, seed)
    if kind == "grid" and nvis * npix > 6e10 or kind == "dropin":
        return None
    s = _inputs(c, seed)
    uvw, freq = s["uvw"], s["freq"]
    dev = uvw.device
    cx, cy = _centre(c)
    if kind == "grid":
        v = s["vis"].to(torch.complex128)
        if s["wgt"] is not None:
            v = v * s["wgt"].double()
        if s["mask"] is not None:
            v = v * s["mask"].double()
        return _dft_image(c, uvw, freq, v, c["nx"], c["ny"], cx, cy)
    if kind == "facets":
        model = torch.zeros((uvw.shape[0], c["nchan"]), dtype=torch.complex128, device=dev)
        for j, q, im in zip(_jobs(c), s["srcs"], s["imgs"]):
            at = torch.nonzero(im)
            lmn = _lmn(c, at[:, 0], at[:, 1], j["npix_x"], j["npix_y"], j["center_x"],
                       j["center_y"], dev)
            ch = slice(j["chan_begin"], j["chan_end"])
            model[:, ch] += _dft_vis(uvw, freq[ch], lmn, im[at[:, 0], at[:, 1]].double())
        if s["wgt"] is not None:
            model *= s["wgt"].double()
        return {"model": model, "images": None}
    im = s["img"]
    at = torch.nonzero(im)
    lmn = _lmn(c, at[:, 0], at[:, 1], c["nx"], c["ny"], cx, cy, dev)
    model = _dft_vis(uvw, freq, lmn, im[at[:, 0], at[:, 1]].double())
    if kind == "predict":
        if s["wgt"] is not None:
            model *= s["wgt"].double()
        if s["mask"] is not None:
            model *= s["mask"].double()
        return model
    if kind == "gradient":
        return {"gradient": None, "model": model}
    n = uvw.shape[0]
    cuts = [n * k // c["nchunk"] for k in range(c["nchunk"] + 1)]
    return {"model": [model[a:b] for a, b in zip(cuts, cuts[1:])], "image": None}


def _exact_weights(c, seed):
    """Briggs weights (robust 0): the weights summed per uv cell of the
    v >= 0 half plane, 1 / (1 + W s^2) with s^2 = 25 sum(W) / sum(W^2)."""
    s = _inputs(c, seed)
    uvw, w = s["uvw"], s["wgt"].double()
    lam = torch.as_tensor(C_LIGHT / s["freq"], device=uvw.device)
    u, v = uvw[:, 0:1] / lam, uvw[:, 1:2] / lam
    u, v = torch.where(v < 0, -u, u), v.abs()
    p = c["pix"] * ARCSEC
    x = torch.floor(u * float(c["nx"]) * p + float(c["nx"] // 2)).long()
    y = torch.floor(v * float(c["ny"]) * p).long()
    ok = (x >= 0) & (x < c["nx"]) & (y < c["ny"] // 2)
    cell = torch.where(ok, x + y * c["nx"], 0)
    wk = torch.where(ok, w, 0.0)
    grid = torch.zeros(c["nx"] * (c["ny"] // 2), dtype=torch.float64, device=uvw.device)
    grid.index_add_(0, cell.reshape(-1), wk.reshape(-1))
    s2 = 25.0 / ((grid * grid).sum() / wk.sum())
    return torch.where(ok, w / (1.0 + grid[cell] * s2), 0.0)
