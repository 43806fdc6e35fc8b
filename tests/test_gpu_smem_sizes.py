"""Every box size runs in a process that has run no larger one before.

A kernel's dynamic and static shared memory together may exceed 48 KB where the dynamic part
alone does not (the warp form of the diagnostics at fit radii of 10 px); a limit that an
earlier, larger launch left behind would hide that.  So the sizes go upwards in a process of
their own: warp and block diagnostics, single-node, gridded and Gaussian stamps.
"""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np
import crowdphot_b200 as cpb
from crowdphot_b200.simulate import moffat_epsf
rng = np.random.default_rng(0)
psf = {KIND}
kind_fixed = {FIXED}
for n, radii in {SIZES}:
    shape = (300, 301) if n > 100 else (90, 101)
    img, iv = rng.normal(0, 3, shape), np.full(shape, 0.1)
    src = dict(y=rng.uniform(1, shape[0], n), x=rng.uniform(1, shape[1], n), flux=rng.uniform(100, 1000, n))
    for r in radii:
        g = cpb.fit_all_stars_simultaneous(img, psf, src, float(r), fixed=kind_fixed, inv_var=iv, model_rad=float(r),
                                           max_iter=1, precision={PREC!r})
        assert np.isfinite(g.residual).all(), r
        if {PREC!r} == "fp64" and r < 14:
            m = cpb.fit_all_stars(img, psf, src, float(r), n_passes=1, fixed=kind_fixed, inv_var=iv, max_iter=2)
            assert np.isfinite(m.residual).all(), r
"""
MANY = (700, [2, 4, 5, 6, 7, 8, 9, 9.5, 10, 10.5, 11, 12, 13])
FEW = (6, list(range(2, 45)))


@pytest.mark.parametrize("kind,fixed", [("moffat_epsf().psfs[0]", {"bkg": 0.0}), ("cpb.GriddedPSFModel([moffat_epsf(fwhm=f).psfs[0] for f in (2.6, 2.8, 2.8, 3.0)], [1.0, 1.0, 300.0, 300.0], "
                                         "[1.0, 300.0, 1.0, 300.0])", {"bkg": 0.0}),
                                        ("cpb.CircularGaussianPSF(fwhm=2.4)", {"bkg": 0.0, "fwhm": 2.4})])
@pytest.mark.parametrize("sizes,prec", [([MANY], "fp64"), ([FEW], "fp64"), ([FEW], "mixed")])
def test_sizes_upwards(kind, fixed, sizes, prec):
    script = SCRIPT.format(KIND=kind, FIXED=fixed, SIZES=sizes, PREC=prec)
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = %r\n" % sys.path + script],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
