"""model_rad = :auto on the device: the noise quantile's radix select against the oracle.

The radii are integers and the device uses the host arithmetic's roundings, so they must
be equal.  Weight images at the edges of the select: every weight the same, two values
(the interpolated order statistics differ), duplicates around the quantile, zeros, NaN and
infinities in the sample, magnitudes over the whole exponent range, a single positive
weight; samples of every pixel and of every fourth; no positive weight is refused.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.simulate import moffat_epsf

pytestmark = pytest.mark.gpu


def weights(kind, shape):
    rng = np.random.default_rng(11)
    w = rng.uniform(0.001, 0.02, shape)
    if kind == "same":
        w[:] = 0.0125
    elif kind == "two":
        w = np.where(rng.random(shape) < 0.84, 0.004, 0.016)
    elif kind == "duplicates":
        w = rng.integers(1, 6, shape) / 256.0
    elif kind == "bad":
        w[rng.random(shape) < 0.3] = 0.0
        w[rng.random(shape) < 0.1] = np.nan
        w[rng.random(shape) < 0.1] = np.inf
        w[rng.random(shape) < 0.1] = -1.0
    elif kind == "range":
        w = 10.0 ** rng.uniform(-300, 2, shape)
        w[rng.random(shape) < 0.5] = 0.01
    elif kind == "one":
        w[:] = 0.0
        w[16, 16] = 0.01
    return w


@pytest.mark.parametrize("shape", [(40, 33), (601, 500)])
@pytest.mark.parametrize("kind", ["uniform", "same", "two", "duplicates", "bad", "range", "one"])
def test_radii_equal_the_oracle(shape, kind):
    from oracle import orc_fit_simultaneous
    if kind == "one" and shape[0] > 100:
        pytest.skip("the sampled pixels of the large image miss the single weight")
    rng = np.random.default_rng(4)
    psf = moffat_epsf()
    n = 12
    src = dict(y=rng.uniform(12, 25, n), x=rng.uniform(12, 25, n), flux=10 ** rng.uniform(0, 6, n))
    img = rng.normal(0, 10, shape)
    w = weights(kind, shape)
    for nsigma, rmax in ((1.0, None), (0.3, 31)):
        kw = dict(fixed={"bkg": 0.0}, inv_var=w, max_iter=1, model_rad_nsigma=nsigma, model_rad_max=rmax, debug=True)
        g = cpb.fit_all_stars_simultaneous(img, psf, src, 4, **kw)
        o = orc_fit_simultaneous(img, psf, src, 4, **kw)
        assert np.array_equal(g.debug["active"], o.debug["active"])
        assert np.array_equal(g.debug["model_R"], o.debug["model_R"])
        if kind == "uniform":
            assert len(set(g.debug["model_R"])) > 3


def test_a_sample_without_positive_weights_is_refused():
    w = np.zeros((600, 600))
    w[301, 300] = 1.0  # keeps a star active; the sampled rows do not hold it
    with pytest.raises(cpb.ArgumentError, match="no positive finite weights"):
        cpb.fit_all_stars_simultaneous(np.zeros((600, 600)), moffat_epsf(), dict(y=[300.0], x=[300.0], flux=[10.0]), 4,
                                       fixed={"bkg": 0.0}, inv_var=w)
