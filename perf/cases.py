"""Timed workloads of the framework, each one pass through a public entry point.

Every case is a plain dict whose "kind" names the call:

  field    fit_all_stars_simultaneous of one image (host arrays in, host arrays out)
  device   the same fit of an image that is on the GPU already (the C entry for device buffers;
           the catalogue of results comes back to host arrays)
  served   several fields submitted to a Server and waited for
  passes   fit_all_stars, the sequential multi-pass photometry of one image
  cutouts  a BatchGraph over device-resident fit_star cutouts, replayed
  groups   a BatchGraph over device-resident blended star groups, replayed
  star     one fit_star call on one cutout of a host image

Inputs are synthetic crowded-field data of the kind the benchmark uses: power-law or
log-uniform fluxes, a Moffat (tabulated at 4x) or Gaussian PSF, a smooth background of 50-200
counts, Poisson and read noise, inverse-variance weights and perturbed initial guesses.  The
catalogues are what detection and deblending list: stars above the noise, a PSF width apart.  They are drawn on the GPU from the seed alone (star images are summed in
fixed point, so the order of the sums does not matter).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crowdphot.jl_b200"))

import crowdphot_b200 as cpb  # noqa: E402
from crowdphot_b200 import _abi  # noqa: E402
from crowdphot_b200.photometry import SimOutputs, _lm_outputs, group_outputs, sim_params  # noqa: E402
from crowdphot_b200.psf import replace_params  # noqa: E402
from crowdphot_b200.simulate import moffat_epsf  # noqa: E402

BETA = 3.0
FWHM = 2.8         # of the tabulated Moffat
GAUSS_FWHM = 2.5
FAINT = 400.0      # counts of the faintest star of a field's catalogue (about 6 sigma: what detection lists)
CELL, SEP = 5, 3   # catalogue stars sit in cells of CELL px, at least SEP px apart (deblended detections)
HALF = 13          # half-width of the rendered star boxes
FIXED = 16777216.0  # fixed-point unit of the star image sums (2^24 a count)


def listed():
    return [
        # one star at a time from a user's own loop: latency only
        dict(name="star_image", kind="star", psf="image", side=25, dtype="float32"),
        # the smallest whole-image call: 256^2 Float64, Gaussian PSF, tight linear tolerance
        dict(name="field_gauss_256", kind="field", psf="gauss", ny=256, nx=256, n=200, dtype="float64", fit_rad=7.0,
             model_rad=7.0, max_iter=20, linear_tol=1e-8, flux="loguniform", precision="fp64", residual=True),
        # an ordinary ragged cutout of a survey image with every default: per-star model radii
        # (:auto), residual image and all diagnostics
        dict(name="field_auto_odd", kind="field", psf="image", ny=613, nx=421, n=1400, dtype="float32", fit_rad=9.0,
             model_rad=0.0, max_iter=40, linear_tol=1e-6, flux="powerlaw", precision="fp64", residual=True),
        # a spatially varying PSF (2 x 2 nodes), as the Roman ePSF grids are used
        dict(name="field_grid_500", kind="field", psf="grid", ny=500, nx=500, n=1500, dtype="float64", fit_rad=8.0,
             model_rad=12.0, max_iter=12, linear_tol=1e-6, flux="loguniform", precision="fp64", residual=True),
        # the crowded field of the benchmark, plain FP64 form
        dict(name="field_crowded_2048", kind="field", psf="image", ny=2048, nx=2048, n=50000, dtype="float32",
             fit_rad=12.0, model_rad=12.0, max_iter=40, linear_tol=1e-6, flux="powerlaw", precision="fp64",
             residual=True),
        # a wide, sparser detector image, catalogue only
        dict(name="device_wide_4096", kind="device", psf="image", ny=4096, nx=4000, n=60000, dtype="float32",
             fit_rad=8.0, model_rad=12.0, max_iter=15, linear_tol=1e-6, flux="powerlaw", precision="fp64",
             residual=False),
        # the mixed-precision form on a crowded field: a Float32-stamp iteration from the catalogue's
        # guesses, then refinement to the Float64 solution
        dict(name="device_mixed_1500", kind="device", psf="image", ny=1500, nx=1501, n=14000, dtype="float32",
             fit_rad=9.0, model_rad=12.0, max_iter=1, linear_tol=1e-6, flux="loguniform", precision="mixed", refine=6,
             residual=False),
        # requests of a photometry service: fields of uneven sizes in flight together
        dict(name="served_six", kind="served", psf="image", ny=512, nx=512, n=6, density=0.008, dtype="float32",
             fit_rad=12.0, model_rad=12.0, max_iter=40, linear_tol=1e-6, flux="powerlaw", precision="fp64",
             residual=False),
        # sequential photometry, three passes over a crowded field
        dict(name="passes_1024", kind="passes", psf="image", ny=1024, nx=1024, n=12500, dtype="float32", fit_rad=12.0,
             passes=3, flux="powerlaw"),
        # large batch of isolated stars of uneven cutouts
        dict(name="cutouts_100k", kind="cutouts", psf="image", n=100000, smin=9, smax=41, dtype="float32"),
        # blends of a few stars each, many at once
        dict(name="groups_4k", kind="groups", psf="image", n=4000, kmin=2, kmax=12, dtype="float32", fit_rad=6.0,
             model_rad=6.0),
        # a handful of blends with a Gaussian PSF in Float64
        dict(name="groups_gauss_60", kind="groups", psf="gauss", n=60, kmin=2, kmax=8, dtype="float64", fit_rad=5.0,
             model_rad=5.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["field", "field", "device", "device", "served", "passes", "cutouts", "groups", "star"])
    dtype = rng.choice(["float32", "float64"])
    if kind == "star":
        return dict(kind="star", psf=rng.choice(["image", "gauss"]), side=rng.randint(9, 41), dtype=dtype)
    if kind == "cutouts":
        smin = rng.randint(9, 21)
        return dict(kind="cutouts", psf=rng.choice(["image", "image", "gauss"]), n=_log_int(rng, 100, 100000),
                    smin=smin, smax=rng.randint(smin, 41), dtype=dtype)
    if kind == "groups":
        kmin, rad = rng.randint(1, 4), float(rng.randint(4, 7))
        return dict(kind="groups", psf=rng.choice(["image", "image", "gauss"]), n=_log_int(rng, 20, 4000), kmin=kmin,
                    kmax=rng.randint(kmin, 12), dtype=dtype, fit_rad=rad, model_rad=rad)
    density = rng.uniform(0.002, 0.012)
    if kind == "served":
        side = _log_int(rng, 200, 700)
        return dict(kind="served", psf="image", ny=side, nx=side, n=rng.randint(2, 8), density=round(density, 5),
                    dtype="float32", fit_rad=float(rng.randint(6, 12)), model_rad=12.0, max_iter=40, linear_tol=1e-6,
                    flux="powerlaw", precision="fp64", residual=False)
    if kind == "passes":
        ny, nx = _log_int(rng, 200, 1100), _log_int(rng, 200, 1100)
        return dict(kind="passes", psf=rng.choice(["image", "image", "gauss"]), ny=ny, nx=nx,
                    n=int(density * ny * nx), dtype=dtype, fit_rad=float(rng.randint(5, 12)), passes=rng.randint(1, 3),
                    flux="powerlaw")
    psf = rng.choice(["image", "image", "image", "gauss", "grid"])
    top = 600 if psf == "grid" else 2000
    ny, nx = _log_int(rng, 200, top), _log_int(rng, 200, top)
    mixed = psf == "image" and rng.random() < 0.25
    density *= 0.5 if mixed else 1.0
    return dict(kind=kind, psf=psf, ny=ny, nx=nx, n=max(20, int(density * ny * nx)), dtype=dtype,
                fit_rad=float(rng.randint(5, 10 if mixed else 12)), model_rad=rng.choice([0.0, 8.0, 12.0]),
                max_iter=1 if mixed else rng.choice([12, 20, 40]), linear_tol=1e-6,
                flux="loguniform" if mixed else rng.choice(["powerlaw", "loguniform"]),
                precision="mixed" if mixed else "fp64",
                refine=6 if mixed else 0, residual=kind == "field" and rng.random() < 0.6)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_psfs = {}


def _psf(kind):
    """The PSF object a program builds once and uses for all its images."""
    if kind not in _psfs:
        if kind == "gauss":
            _psfs[kind] = cpb.CircularGaussianPSF(fwhm=GAUSS_FWHM)
        elif kind == "image":
            _psfs[kind] = moffat_epsf(fwhm=FWHM)
        else:
            nodes = [moffat_epsf(fwhm=f, size=121).psfs[0] for f in (2.6, 2.8, 2.8, 3.0)]
            _psfs[kind] = cpb.GriddedPSFModel(nodes, [1.0, 1.0, 600.0, 600.0], [1.0, 600.0, 1.0, 600.0])
    return _psfs[kind]


def _fixed(kind):
    return {"fwhm": GAUSS_FWHM, "bkg": 0.0} if kind == "gauss" else {"bkg": 0.0}


def _moffat(r2, fwhm):
    a2 = (fwhm / 2) ** 2 / (2 ** (1 / BETA) - 1)
    return (BETA - 1) / (math.pi * a2) * (1 + r2 / a2) ** (-BETA)


def _profile(kind, dy, dx, y, x):
    """Unit-flux profile at pixel offsets (dy, dx) of stars at (y, x)."""
    r2 = dy * dy + dx * dx
    if kind == "gauss":
        s = 4 * math.log(2) / GAUSS_FWHM ** 2
        return s / math.pi * torch.exp(-s * r2)
    if kind == "image":
        return _moffat(r2, FWHM) * ((dy.abs() <= 12.5) & (dx.abs() <= 12.5))
    v, u = ((y - 1) / 599).clamp(0, 1), ((x - 1) / 599).clamp(0, 1)
    return (1 - v) * (1 - u) * _moffat(r2, 2.6) + (v + u - 2 * u * v) * _moffat(r2, 2.8) + v * u * _moffat(r2, 3.0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _uniform(g, lo, hi, n):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, n):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _places(g, ny, nx, n):
    """n positions in distinct CELL px cells of the field, SEP px apart at least (fewer than n where
    the field has not so many cells)."""
    my, mx = (ny - 1) // CELL, (nx - 1) // CELL
    cell = torch.randperm(my * mx, generator=g, device="cuda")[:n]
    room = float(CELL - SEP)
    y = 1 + CELL * (cell % my) + 0.5 * SEP + _uniform(g, 0.0, room, cell.numel())
    x = 1 + CELL * torch.div(cell, my, rounding_mode="floor") + 0.5 * SEP + _uniform(g, 0.0, room, cell.numel())
    return y, x


def _fluxes(g, how, n):
    u = _uniform(g, 0.0, 1.0, n)
    if how == "loguniform":
        return torch.exp(math.log(FAINT) + u * math.log(1e5 / FAINT))
    lo, hi = FAINT ** -0.5, 1e6 ** -0.5  # dN/dF ~ F^-1.5
    return (lo + u * (hi - lo)) ** -2


def _noisy(g, model, bkg):
    """Poisson and read noise on model + bkg, and the inverse variances."""
    img = torch.poisson(model + bkg, generator=g) + 5.0 * torch.randn(model.shape, generator=g, device="cuda",
                                                                        dtype=torch.float64)
    return img, 1.0 / (model + bkg + 25.0)


def _stars_image(kind, ny, nx, y, x, f):
    """Sum of star images on an ny x nx field, stored (nx, ny) (the column-major image)."""
    total = torch.zeros(nx * ny, dtype=torch.int64, device="cuda")
    off = torch.arange(-HALF, HALF + 1, device="cuda", dtype=torch.float64)
    for c in range(0, y.numel(), 16384):
        yc, xc, fc = (a[c:c + 16384, None, None] for a in (y, x, f))
        gy = yc.round() + off[None, None, :]
        gx = xc.round() + off[None, :, None]
        val = (fc * _profile(kind, gy - yc, gx - xc, yc, xc) * FIXED).round().to(torch.int64)
        at = ((gx - 1) * ny + (gy - 1)).to(torch.int64)
        keep = (gy >= 1) & (gy <= ny) & (gx >= 1) & (gx <= nx)
        total.index_add_(0, at[keep], val[keep])
    return (total.to(torch.float64) / FIXED).reshape(nx, ny)


def _field(kind, ny, nx, n, how, dtype, seed):
    """(image, background, inv_var, sources) as host arrays, images column-major."""
    g = _gen(seed)
    y, x = _places(g, ny, nx, n)
    n = y.numel()
    f = _fluxes(g, how, n)
    model = _stars_image(kind, ny, nx, y, x, f)
    u = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None] / max(nx - 1, 1)
    v = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :] / max(ny - 1, 1)
    bkg = 50.0 + 150.0 * (0.6 * u + 0.4 * v * v)
    img, iv = _noisy(g, model, bkg)
    src = dict(y=y + 0.3 * _normal(g, n), x=x + 0.3 * _normal(g, n), flux=f * _uniform(g, 0.9, 1.1, n))
    host = lambda t: t.to(getattr(torch, dtype)).cpu().numpy().T  # noqa: E731
    return host(img), host(bkg), host(iv), {k: t.cpu().numpy() for k, t in src.items()}


def _snr_flux(g, kind, n):
    """Fluxes whose signal to noise is log-uniform in 5-1000 over background and read noise."""
    snr = torch.exp(math.log(5.0) + _uniform(g, 0.0, 1.0, n) * math.log(200.0))
    a2 = (FWHM / 2) ** 2 / (2 ** (1 / BETA) - 1)
    area = math.pi * GAUSS_FWHM ** 2 / (2 * math.log(2)) if kind == "gauss" else \
        math.pi * a2 * (2 * BETA - 1) / (BETA - 1) ** 2
    return (snr ** 2 + torch.sqrt(snr ** 4 + 4 * snr ** 2 * area * 125.0)) / 2


def _cutouts(case, seed):
    g = _gen(seed)
    n, kind, dt = case["n"], case["psf"], getattr(torch, case["dtype"])
    ny = torch.randint(case["smin"], case["smax"] + 1, (n,), generator=g, device="cuda")
    nx = torch.randint(case["smin"], case["smax"] + 1, (n,), generator=g, device="cuda")
    y1 = torch.randint(1, 4000, (n,), generator=g, device="cuda")
    x1 = torch.randint(1, 4000, (n,), generator=g, device="cuda")
    y = y1 + (ny - 1) / 2 + _uniform(g, -0.5, 0.5, n)
    x = x1 + (nx - 1) / 2 + _uniform(g, -0.5, 0.5, n)
    f = _snr_flux(g, kind, n)
    size = ny * nx
    off = torch.cumsum(size, 0) - size
    c = torch.repeat_interleave(torch.arange(n, device="cuda"), size)
    e = torch.arange(c.numel(), device="cuda") - off[c]
    dy = (y1[c] + e % ny[c]) - y[c]
    dx = (x1[c] + torch.div(e, ny[c], rounding_mode="floor")) - x[c]
    img, iv = _noisy(g, f[c] * _profile(kind, dy, dx, y[c], x[c]), 100.0)
    par = [y + 0.3 * _normal(g, n), x + 0.3 * _normal(g, n), f * _uniform(g, 0.9, 1.1, n), torch.zeros_like(f)]
    if kind == "gauss":
        par.insert(2, torch.full_like(f, GAUSS_FWHM))
    i32 = lambda t: t.to(torch.int32)  # noqa: E731
    return dict(offsets=off, ny=i32(ny), nx=i32(nx), y1=i32(y1), x1=i32(x1), pix=(img - 100.0).to(dt),
                inv_var=iv.to(dt), init=torch.stack(par, 1).contiguous())


def _groups(case, seed):
    g = _gen(seed)
    n, kind, dt = case["n"], case["psf"], getattr(torch, case["dtype"])
    k = case["kmin"] + torch.randperm(n, generator=g, device="cuda") % (case["kmax"] - case["kmin"] + 1)
    side = 8 * k + 17
    size = side * side
    off = torch.cumsum(size, 0) - size
    so = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    so[1:] = torch.cumsum(k, 0)
    grp = torch.repeat_interleave(torch.arange(n, device="cuda"), k)
    ns = grp.numel()
    # the k stars of a group in k stripes of its columns, SEP px apart at least, 2 px inside the cutout
    stripe = (side[grp] - 5.0) / k[grp]
    i = torch.arange(ns, device="cuda") - so[:-1][grp]
    y = 3 + (side[grp] - 5) * _uniform(g, 0.0, 1.0, ns)
    x = 3 + stripe * i + 0.5 * SEP + (stripe - SEP) * _uniform(g, 0.0, 1.0, ns)
    f = _snr_flux(g, kind, ns)
    total = torch.zeros(int(size.sum()), dtype=torch.int64, device="cuda")
    d = torch.arange(-HALF, HALF + 1, device="cuda", dtype=torch.float64)
    for c in range(0, ns, 16384):
        yc, xc, fc, sd, oc = (a[c:c + 16384, None, None] for a in (y, x, f, side[grp], off[grp]))
        gy = yc.round() + d[None, None, :]
        gx = xc.round() + d[None, :, None]
        val = (fc * _profile(kind, gy - yc, gx - xc, yc, xc) * FIXED).round().to(torch.int64)
        at = oc + ((gx - 1) * sd + (gy - 1)).to(torch.int64)
        keep = (gy >= 1) & (gy <= sd) & (gx >= 1) & (gx <= sd)
        total.index_add_(0, at[keep], val[keep])
    img, iv = _noisy(g, total.to(torch.float64) / FIXED, 100.0)
    i32 = lambda t: t.to(torch.int32)  # noqa: E731
    return dict(offsets=off, ny=i32(side), nx=i32(side), pix=(img - 100.0).to(dt), inv_var=iv.to(dt),
                star_offsets=so, y=y + 0.3 * _normal(g, ns), x=x + 0.3 * _normal(g, ns),
                flux=f * _uniform(g, 0.9, 1.1, ns))


def _field_kw(case, bkg, iv):
    kw = dict(fixed=_fixed(case["psf"]), inv_var=iv, background=bkg, max_iter=case["max_iter"],
              linear_tol=case["linear_tol"], precision=case["precision"], refine_iters=case.get("refine", 0),
              residual=case["residual"])
    if case["model_rad"] > 0:
        kw["model_rad"] = case["model_rad"]
    return kw


def prepare(case, seed):
    kind, psf = case["kind"], _psf(case["psf"])
    if kind == "field":
        img, bkg, iv, src = _field(case["psf"], case["ny"], case["nx"], case["n"], case["flux"], case["dtype"], seed)
        return dict(kind=kind, args=(img, psf, src, case["fit_rad"]), kw=_field_kw(case, bkg, iv))
    if kind == "device":
        img, bkg, iv, src = _field(case["psf"], case["ny"], case["nx"], case["n"], case["flux"], case["dtype"], seed)
        kw = _field_kw(case, None, None)
        fixed = kw.pop("fixed")
        for k in ("inv_var", "background", "residual"):
            kw.pop(k)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()  # noqa: E731
        keep = [up(a) for a in (img, iv, bkg)] + [up(src[k]) for k in ("y", "x", "flux")]
        outs = SimOutputs(src["y"].size, case["ny"], case["nx"], 0, residual=False)
        ctx = cpb.get_context()
        ptr = [C.c_void_p(t.data_ptr()) for t in keep]
        params = sim_params(psf, case["fit_rad"], fixed, inv_var_given=True, **kw)
        item = _abi.CPB_F32 if case["dtype"] == "float32" else _abi.CPB_F64
        args = (ctx.handle, ctx.psf_handle(psf), C.byref(params), ptr[0], item, case["ny"], case["nx"], ptr[1], ptr[2],
                src["y"].size, *ptr[3:], C.byref(outs.c))
        return dict(kind=kind, ctx=ctx, keep=(keep, params), outs=outs, args=args)
    if kind == "served":
        calls = []
        for i in range(case["n"]):  # sides from the given one down to half of it, and twice that for one in three
            ny = case["ny"] * (2 if i % 3 == 1 else 1) - 17 * i
            nx = case["nx"] * (2 if i % 3 == 1 else 1) - 31 * i // 2
            img, bkg, iv, src = _field(case["psf"], ny, nx, int(case["density"] * ny * nx), case["flux"],
                                       case["dtype"], 1000 * seed + i)
            calls.append(((img, psf, src, case["fit_rad"]), _field_kw(case, bkg, iv)))
        server = cpb.Server(max_inflight=4)
        server.psf_id(psf)
        return dict(kind=kind, server=server, calls=calls)
    if kind == "passes":
        img, bkg, iv, src = _field(case["psf"], case["ny"], case["nx"], case["n"], case["flux"], case["dtype"], seed)
        return dict(kind=kind, args=(img - bkg, psf, src, case["fit_rad"]),
                    kw=dict(n_passes=case["passes"], fixed=_fixed(case["psf"]), inv_var=iv))
    if kind == "star":
        g = _gen(seed)
        s = case["side"]
        y, x = (s + 1 + _uniform(g, -0.5, 0.5, 1) for _ in range(2))
        f = _snr_flux(g, case["psf"], 1) + 2000.0
        img, iv = _noisy(g, _stars_image(case["psf"], 2 * s + 1, 2 * s + 1, y, x, f), 100.0)
        lo = s + 1 - s // 2
        host = lambda t: t.to(getattr(torch, case["dtype"])).cpu().numpy().T  # noqa: E731
        start = dict(y=float(y) + 0.2, x=float(x) - 0.2, flux=1.05 * float(f))
        node = psf if case["psf"] == "gauss" else psf.psfs[0]
        return dict(kind=kind, args=(replace_params(node, **start), host(img - 100.0), ((lo, lo + s - 1),) * 2),
                    kw=dict(fixed=_fixed(case["psf"]), inv_var=host(iv)))
    cuda = lambda o: {k: torch.from_numpy(v).cuda() for k, v in o.items()}  # noqa: E731
    if kind == "cutouts":
        lm = _cutouts(case, seed)
        lm["out"] = cuda(_lm_outputs(case["n"], lm["init"].shape[1], 3))
        graph = cpb.BatchGraph(psf, lm=lm, lm_fixed=_fixed(case["psf"]), autotune=0)
        return dict(kind=kind, graph=graph, out=lm["out"])
    gr = _groups(case, seed)
    gr["out"] = cuda(group_outputs(gr["y"].numel(), case["n"]))
    graph = cpb.BatchGraph(psf, groups=gr, fit_rad=case["fit_rad"], autotune=0,
                           group_kw=dict(fixed=_fixed(case["psf"]), model_rad=case["model_rad"]))
    return dict(kind=kind, graph=graph, out=gr["out"])


# ---------------------------------------------------------------------------
# passes
# ---------------------------------------------------------------------------
_FIELDS = ("y", "x", "flux", "y_err", "x_err", "flux_err", "chisq", "qfit", "qfit_expected", "qfit_z", "crowding",
           "spread_model", "spread_model_err", "converged", "valid", "n_iter")


def _arrays(r, residual):
    out = {k: getattr(r, k) for k in _FIELDS}
    if residual:
        out["residual"] = r.residual
    return out


def run(state):
    kind = state["kind"]
    if kind == "field":
        return _arrays(cpb.fit_all_stars_simultaneous(*state["args"], **state["kw"]), state["kw"]["residual"])
    if kind == "device":
        ctx, outs = state["ctx"], state["outs"]
        ctx.raise_for(ctx.lib.cpb_fit_simultaneous_device(*state["args"]), "cpb_fit_simultaneous_device")
        return {k: getattr(outs, k) for k in _FIELDS}
    if kind == "served":
        pending = [state["server"].submit(*a, **kw) for a, kw in state["calls"]]
        done = [r.result() for r in pending]
        return {k: np.concatenate([getattr(r, k) for r in done]) for k in _FIELDS}
    if kind == "passes":
        return _arrays(cpb.fit_all_stars(*state["args"], **state["kw"]), True)
    if kind == "star":
        best, res = cpb.fit_star(*state["args"], **state["kw"])
        return dict(y=best.y, x=best.x, flux=best.flux, cov=res.cov, cost=res.minimum, cost_init=res.cost_init,
                    chisq=res.chisq, iterations=res.iterations, converged=res.converged)
    state["graph"].launch()
    return {k: v for k, v in state["out"].items() if k != "sigma_final"}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: inputs read once and results written once.  Flops: the least-squares iterations at
    nominal counts (a star settles in about six outer iterations of ten inner ones each; a
    cutout's fit in six evaluations), with 100 operations a profile evaluation with derivatives,
    30 a value and 12 a pixel of an inner iteration."""
    item = 4 if case["dtype"] == "float32" else 8
    kind = case["kind"]
    if kind == "star":
        px = case["side"] ** 2
        return dict(bytes=2.0 * item * px + 200, flops=6.0 * 120 * px)
    if kind == "cutouts":
        px = case["n"] * (0.5 * (case["smin"] + case["smax"])) ** 2
        return dict(bytes=2.0 * item * px + 300.0 * case["n"], flops=6.0 * 120 * px)
    box = (2 * math.ceil(case["fit_rad"]) + 1) ** 2
    if kind == "passes":
        px = case["ny"] * case["nx"]
        return dict(bytes=px * (2.0 * item + 8) + 170.0 * case["n"],
                    flops=case["passes"] * case["n"] * box * (5.0 * 120 + 60))
    outer = min(case.get("max_iter", 40) + case.get("refine", 0), 6)
    model = (2 * math.ceil(case["model_rad"] or case["fit_rad"]) + 1) ** 2
    star = outer * (box * (100 + 10 * 12.0) + 2 * model * 30)
    if kind == "groups":
        k = 0.5 * (case["kmin"] + case["kmax"])
        return dict(bytes=case["n"] * (2.0 * item * (8 * k + 17) ** 2 + 140 * k), flops=case["n"] * k * star)
    if kind == "served":
        px = case["n"] * case["ny"] * case["nx"] * 2.0
        n = case["density"] * px
    else:
        px, n = float(case["ny"] * case["nx"]), case["n"]
    return dict(bytes=px * (3.0 * item + (8 if case["residual"] else 0)) + 150.0 * n, flops=n * star)


def exact(case, seed):
    """The starting cost of one fit_star call, sum(weight * (model - data)^2) over the cutout at the
    starting parameters.  The other outputs are iterates of a damped least-squares solution stopped
    by its own tolerances: they have no value that could be written down without the iteration."""
    if case["kind"] != "star" or case["psf"] != "gauss":
        return None
    s = prepare(case, seed)
    model, img, ((ya, yb), (xa, xb)) = s["args"]
    d = img[ya - 1:yb, xa - 1:xb].astype(np.float64)
    w = s["kw"]["inv_var"][ya - 1:yb, xa - 1:xb].astype(np.float64)
    py, px = np.meshgrid(np.arange(ya, yb + 1.0), np.arange(xa, xb + 1.0), indexing="ij")
    c = 4 * math.log(2) / GAUSS_FWHM ** 2
    m = model.flux * c / math.pi * np.exp(-c * ((py - model.y) ** 2 + (px - model.x) ** 2))
    return dict(y=None, x=None, flux=None, cov=None, cost=None, cost_init=float(np.sum(w * (m - d) ** 2)), chisq=None,
                iterations=None, converged=None)
