"""The shared-memory stamp kernel of single-node ePSFs (k_eval_node) against the oracle.

Sizes where it can go wrong: oversampling 1-5, different on the axes; box half-widths on
either side of the 8 / 16 / 32 lanes a column (R = 3, 4, 7, 8, 15, 16); odd image heights;
boxes cut by the image's edges and by the 32-pixel regions; stars at whole pixels whose
stencils hit the first and the last table sample exactly; fewer free parameters; a model
box wider than the fit box; one star.  A table of unstructured values shows any
misplaced sample.

Tolerance: both sides compute in FP64, a few hundred terms a sum, on separated stars
(normal matrices with a condition number below 1e4): rounding differences stay below
1e-11 relative, and 1e-9 is asked for.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb

pytestmark = pytest.mark.gpu


def table_psf(size, os_, seed):
    rng = np.random.default_rng(seed)
    ny, nx = size
    sx, sy = os_
    y = (np.arange(ny) - (ny - 1) / 2) / sy
    x = (np.arange(nx) - (nx - 1) / 2) / sx
    g = np.exp(-(y[:, None] ** 2 + x[None, :] ** 2) / 4.0) + 0.02
    return cpb.ImagePSF(g * (1 + 0.05 * rng.random((ny, nx))), oversampling=os_, normalize=True)


@pytest.mark.parametrize("size,os_,R,model_rad,shape,fixed", [
    ((33, 33), (4, 4), 5, 5, (97, 64), {}),        # ends hit at whole pixels (grid half-width 4 px)
    ((33, 17), (2, 4), 8, 8, (61, 75), {}),
    ((31, 41), (5, 3), 4, 4, (50, 41), {}),
    ((25, 25), (1, 1), 7, 9, (64, 63), {}),
    ((101, 101), (4, 4), 12, 12, (99, 70), {}),
    ((101, 101), (4, 4), 3, 3, (40, 40), {}),
    ((101, 101), (4, 4), 15, 15, (67, 90), {}),
    ((64, 90), (3, 2), 16, 16, (66, 81), {}),      # 33 px boxes: 17 granules a column
    ((101, 101), (4, 4), 6, 16, (70, 70), {"flux": 800.0}),
])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fields_match_the_oracle(size, os_, R, model_rad, shape, fixed, precision):
    from oracle import orc_fit_simultaneous
    psf = table_psf(size, os_, seed=size[0] + 7 * R)
    rng = np.random.default_rng(R + size[1])
    ny, nx = shape
    # whole-pixel and sub-pixel guesses, one at every edge
    ys = np.array([1.0, ny, 16.0, 32.0, 33.0, ny / 2 + 0.25])
    xs = np.array([nx / 2, 20.0, 1.0, nx, 32.0, 10.4])
    truth = dict(y=ys + rng.uniform(-0.15, 0.15, 6), x=xs + rng.uniform(-0.15, 0.15, 6), flux=np.full(6, 800.0))
    from crowdphot_b200.simulate import image_psf_eval
    img = np.zeros(shape)
    gy, gx = np.meshgrid(np.arange(1.0, ny + 1), np.arange(1.0, nx + 1), indexing="ij")
    for y, x, f in zip(truth["y"], truth["x"], truth["flux"]):
        img += f * image_psf_eval(psf, y, x, gy, gx)
    img += rng.normal(0, 1, shape)
    iv = np.where(rng.random(shape) < 0.02, 0.0, rng.uniform(0.5, 2.0, shape))
    init = dict(y=ys, x=xs, flux=np.full(6, 760.0))
    kw = dict(fixed={"bkg": 0.0, **fixed}, inv_var=iv, model_rad=model_rad, max_iter=2, debug=True)
    if precision == "mixed":  # Float32 stamps for one iteration, then FP64 from its parameters
        kw.update(max_iter=1)
    g = cpb.fit_all_stars_simultaneous(img, psf, init, R, precision=precision, **kw)
    o = orc_fit_simultaneous(img, psf, init, R, **kw)
    assert np.array_equal(g.debug["active"], o.debug["active"])
    # Float32 stamps and pixel vectors carry 2^-24 relative errors into the step
    tol = 1e-9 if precision == "fp64" else 3e-5
    for k in ("y", "x", "flux"):
        np.testing.assert_allclose(getattr(g, k), getattr(o, k), rtol=tol, atol=tol)
    for k in ("y_err", "x_err", "flux_err"):
        np.testing.assert_allclose(getattr(g, k), getattr(o, k), rtol=10 * tol, atol=1e-12)
    np.testing.assert_allclose(g.residual, o.residual, rtol=0, atol=800 * tol)


def test_one_star_and_a_node_too_large_for_shared_memory():
    """One star uses one SM; a 401 x 401 node stays with the general kernel: both equal the oracle."""
    from oracle import orc_fit_simultaneous
    rng = np.random.default_rng(5)
    for size, os_ in (((41, 41), (4, 4)), ((401, 401), (4, 4))):
        psf = table_psf(size, os_, seed=3)
        img = rng.normal(10.0, 1.0, (45, 37))
        kw = dict(fixed={"bkg": 0.0}, inv_var=np.ones((45, 37)), model_rad=9, max_iter=2)
        init = dict(y=[20.3], x=[18.6], flux=[500.0])
        g = cpb.fit_all_stars_simultaneous(img, psf, init, 7, **kw)
        o = orc_fit_simultaneous(img, psf, init, 7, **kw)
        for k in ("y", "x", "flux", "flux_err", "residual"):
            np.testing.assert_allclose(getattr(g, k), getattr(o, k), rtol=1e-9, atol=1e-9)
