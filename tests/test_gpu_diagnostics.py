"""The diagnostics of large catalogues (a warp a star, the disk in register lines) against the oracle.

More than four stars an SM, so that the warp form runs; fit radii on either side of its
largest box (28 px: kh = 13 in, kh = 14 out), boxes cut by every edge, stars whose box is
one column wide; single-node, gridded and Gaussian PSFs.  Tolerances: parameters agree to
1e-8 as the fits' tests ask; the diagnostics are sums of up to 800 FP64 terms of those
(1e-7 of a term's scale at most): 1e-6 relative, 1e-8 absolute for spread_model, a
difference of two ratios near one.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.simulate import moffat_epsf, psf_value

pytestmark = pytest.mark.gpu


def scene(kind, seed, side=27, step=11):
    rng = np.random.default_rng(seed)
    g = moffat_epsf()
    psf = cpb.CircularGaussianPSF(fwhm=2.4) if kind == "gauss" else (g.psfs[0] if kind == "image" else g)
    node = cpb.GriddedPSFModel([g.psfs[0]], [0.0], [0.0]) if kind == "image" else psf
    ny, nx = side * step, side * step + 3
    iy, ix = np.divmod(np.arange(side * side), side)
    # the first row and column on the image's edge, the last beyond what the grid covers
    y = 1.0 + iy * step + rng.uniform(-0.3, 0.3, side * side)
    x = 1.0 + ix * step + rng.uniform(-0.3, 0.3, side * side)
    flux = rng.uniform(2e3, 2e4, side * side)
    img = rng.normal(0, 3.0, (ny, nx))
    for a, b, f in zip(y, x, flux):
        y0, y1 = max(int(a) - 12, 1), min(int(a) + 12, ny)
        x0, x1 = max(int(b) - 12, 1), min(int(b) + 12, nx)
        yy, xx = np.meshgrid(np.arange(y0, y1 + 1.0), np.arange(x0, x1 + 1.0), indexing="ij")
        img[y0 - 1:y1, x0 - 1:x1] += psf_value(node, a, b, f, yy, xx)
    iv = np.where(rng.random((ny, nx)) < 0.01, 0.0, rng.uniform(0.05, 0.2, (ny, nx)))
    init = dict(y=y + rng.uniform(-0.1, 0.1, y.size), x=x + rng.uniform(-0.1, 0.1, y.size), flux=0.95 * flux)
    return psf, img, iv, init


KEYS = ("qfit", "qfit_expected", "qfit_z", "crowding", "spread_model_err")


@pytest.mark.parametrize("kind,fit_rad,dtype", [("image", 13.0, np.float32), ("image", 13.5, np.float64),
                                                ("gridded", 6.3, np.float64), ("gauss", 3.0, np.float32)])
def test_multipass_diagnostics_match_the_oracle(kind, fit_rad, dtype):
    from oracle import orc_fit_all_stars
    psf, img, iv, init = scene(kind, 7 + int(fit_rad))
    args = (img.astype(dtype), psf, init, fit_rad)
    kw = dict(n_passes=1, fixed={"bkg": 0.0}, inv_var=iv.astype(dtype), max_iter=60)
    g, o = cpb.fit_all_stars(*args, **kw), orc_fit_all_stars(*args, **kw)
    assert g.valid.sum() > 600 and np.array_equal(g.valid, o.valid)
    ok = g.valid & (g.n_iter == o.n_iter)
    assert ok.sum() >= 0.99 * g.valid.sum()
    for k in KEYS:
        np.testing.assert_allclose(getattr(g, k)[ok], getattr(o, k)[ok], rtol=1e-6, atol=1e-10, err_msg=k)
    np.testing.assert_allclose(g.spread_model[ok], o.spread_model[ok], rtol=1e-6, atol=1e-8)


@pytest.mark.parametrize("kind,fit_rad", [("image", 4.0), ("gridded", 13.0), ("image", 14.0), ("gauss", 5.2)])
def test_simultaneous_diagnostics_match_the_oracle(kind, fit_rad):
    from oracle import orc_fit_simultaneous
    psf, img, iv, init = scene(kind, 50 + int(fit_rad))
    args = (img, psf, init, fit_rad)
    fixed = {"bkg": 0.0, "fwhm": 2.4} if kind == "gauss" else {"bkg": 0.0}
    kw = dict(fixed=fixed, inv_var=iv, model_rad=fit_rad, max_iter=3)
    g, o = cpb.fit_all_stars_simultaneous(*args, **kw), orc_fit_simultaneous(*args, **kw)
    assert g.valid.sum() > 600 and np.array_equal(g.valid, o.valid)
    ok = g.valid
    for k in KEYS:
        np.testing.assert_allclose(getattr(g, k)[ok], getattr(o, k)[ok], rtol=1e-6, atol=1e-10, err_msg=k)
    np.testing.assert_allclose(g.spread_model[ok], o.spread_model[ok], rtol=1e-6, atol=1e-8)
