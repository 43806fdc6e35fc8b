"""The group kernel's forms against the oracle, group by group.

Batches large enough for the half-SM layout and its deferred groups: tight blends (union
far below the bound), stars side by side (union at the bound: deferred), stars far apart
(bounding box beyond the bit map: sorted), images of one row, one column and the box's
own size, boxes cut by every edge, groups of one star, more than 32 stars; model radius
equal to and above the fit half-width; single-node tables whose stencils end inside the
box, gridded and Gaussian PSFs; fewer free parameters; every block size of a bound batch.
Tolerances: the batched groups' parity bar (test_gpu_groups).
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200 import GriddedPSFModel
from crowdphot_b200.simulate import moffat_epsf, psf_value
from test_gpu_groups import compare, run_batch
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu


def pack(psf, groups, dtype, seed):
    """groups: (ny, nx, y, x, flux) each."""
    rng = np.random.default_rng(seed)
    node = GriddedPSFModel([psf], [0.0], [0.0]) if isinstance(psf, cpb.ImagePSF) else psf
    pix, iv, off, cat = [], [], [0], []
    for ny, nx, y, x, f in groups:
        img = rng.normal(0, 1.0, (ny, nx))
        for a, b, c in zip(y, x, f):
            y0, y1, x0, x1 = max(int(a) - 14, 1), min(int(a) + 14, ny), max(int(b) - 14, 1), min(int(b) + 14, nx)
            if y1 < y0 or x1 < x0:
                continue
            yy, xx = np.meshgrid(np.arange(y0, y1 + 1.0), np.arange(x0, x1 + 1.0), indexing="ij")
            img[y0 - 1:y1, x0 - 1:x1] += psf_value(node, a, b, c, yy, xx)
        w = np.where(rng.random((ny, nx)) < 0.02, 0.0, rng.uniform(0.5, 1.5, (ny, nx)))
        pix.append(img.ravel(order="F").astype(dtype))
        iv.append(w.ravel(order="F").astype(dtype))
        off.append(off[-1] + ny * nx)
        cat.append((y + rng.uniform(-0.1, 0.1, len(y)), x + rng.uniform(-0.1, 0.1, len(y)), 0.95 * f))
    n = [len(g[2]) for g in groups]
    j = lambda k: np.concatenate([c[k] for c in cat])
    return dict(pix=np.concatenate(pix), inv_var=np.concatenate(iv), offsets=np.array(off[:-1], np.int64),
                ny=np.array([g[0] for g in groups], np.int32), nx=np.array([g[1] for g in groups], np.int32),
                star_offsets=np.r_[0, np.cumsum(n)].astype(np.int64), y=j(0), x=j(1), flux=j(2))


def shapes(seed, R, kmax, apart=False):
    rng = np.random.default_rng(seed)
    out = []

    def group(ny, nx, y, x):
        out.append((ny, nx, np.asarray(y, float), np.asarray(x, float), rng.uniform(2e3, 8e3, len(y))))
    k = kmax
    side = 2 * R + 6 * int(np.ceil(np.sqrt(k)))
    for _ in range(3):   # tight blends on a jittered grid
        g = np.arange(k)
        group(side + 1, side, R + 5 * (g // 4) + rng.uniform(-.4, .4, k), R + 5 * (g % 4) + rng.uniform(-.4, .4, k))
    s = 2 * R + 2        # side by side: no pixel shared, union at the bound
    g = np.arange(k)
    group(s * 3 + 3, s * ((k + 2) // 3) + 3, R + 1 + s * (g % 3) + 0.2, R + 1 + s * (g // 3) - 0.3)
    if apart:            # the corners of an image beyond the bit map
        group(901, 700, [R + 1.2, 900.0 - R, R + 2.0], [R + 1.0, R + 3.3, 699.0 - R])
    group(2 * R + 1, 2 * R + 1, [R + 1.1], [R + 0.9])
    group(1, 23, [1.0], [11.4])
    group(29, 1, [14.3], [1.0])
    group(40, 33, [1.0, 40.0, 20.3, 8.0], [16.0, 16.6, 1.0, 33.0])   # every edge
    return out


@pytest.mark.parametrize("kind,R,model_rad,kmax,dtype,fixed", [
    ("table", 6, 6, 12, np.float32, {}),
    ("table", 6, 9, 12, np.float64, {}),
    ("short", 8, 8, 9, np.float32, {}),        # a table of half-width 4 px inside 17 px boxes
    ("table", 5, 5, 40, np.float64, {}),       # more than 32 stars
    ("table", 7, 7, 12, np.float64, {"flux": 5e3}),
    ("gridded", 6, 6, 12, np.float32, {}),
    ("gauss", 5, 8, 12, np.float64, {}),
])
def test_forms_match_the_oracle(kind, R, model_rad, kmax, dtype, fixed):
    psf = {"table": lambda: table_psf((81, 81), (4, 4), 3), "short": lambda: table_psf((33, 25), (4, 3), 4),
           "gridded": moffat_epsf, "gauss": lambda: cpb.CircularGaussianPSF(fwhm=2.6)}[kind]()
    d = pack(psf, shapes(R + kmax, R, kmax, apart=True), dtype, seed=kmax)
    fx = {"bkg": 0.0, **({"fwhm": 2.6} if kind == "gauss" else {}), **fixed}
    kw = dict(fixed=fx, model_rad=model_rad, max_iter=12)
    out = run_batch(psf, d, R, residual=True, **kw)
    assert out["n_kernel_groups"] + out["n_routed_groups"] == len(d["ny"])
    compare(d, out, psf, R, min_same=0.8, **kw)


def test_the_layouts_give_the_same_bits():
    """A group's result does not depend on the launch that fits it: alone, in a batch whose largest group
    makes it run in the half-SM layout, and deferred from there."""
    psf = table_psf((81, 81), (4, 4), 3)
    gs = shapes(2, 6, 12)
    d = pack(psf, gs, np.float32, seed=1)
    kw = dict(fixed={"bkg": 0.0}, model_rad=6, max_iter=12)
    both = run_batch(psf, d, 6, **kw)
    for g in range(len(gs)):
        s0, s1, o = d["star_offsets"][g], d["star_offsets"][g + 1], d["offsets"][g]
        n = int(d["ny"][g]) * int(d["nx"][g])
        one = dict(pix=d["pix"][o:o + n], inv_var=d["inv_var"][o:o + n], offsets=np.zeros(1, np.int64),
                   ny=d["ny"][g:g + 1], nx=d["nx"][g:g + 1], star_offsets=np.array([0, s1 - s0], np.int64),
                   y=d["y"][s0:s1], x=d["x"][s0:s1], flux=d["flux"][s0:s1])
        r = run_batch(psf, one, 6, **kw)
        if one["star_offsets"][1] < 6:
            continue   # alone these run in smaller blocks, whose sums have another order
        for k in ("y", "x", "flux", "y_err", "chisq", "qfit"):
            np.testing.assert_array_equal(r[k], both[k][s0:s1], err_msg=f"{g} {k}")
