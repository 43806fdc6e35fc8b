"""fit_all_stars keeps the roundings of its chained fits.

Each star is fitted on what the stars before it left of the image, so a rounding in a bright
star's model is in the data of every star it touches, and the quantities divided by a flux
that ends near zero enlarge it.  On these two scenes (fluxes over four decades, two stars in
five listed where there is none) constant cubic weights, scaled derivatives and a reciprocal
solve in place of the per-pixel differences and divisions moved qfit by 4e-8 and 2e-8 of its
norm.

The expected values are this library's own, from a build of commit f07484b on a B200; the
inputs use only additions, multiplications, divisions and uniform draws, so that every host
makes the same bits.  Tolerance: 1e-9 of the norm, what FP64 outputs are held to.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb

pytestmark = pytest.mark.gpu
NY, NX, N = 48, 40, 40


def profile(r2):
    t = 1.0 + r2 / 4.0
    return 0.2546 / (t * t * t)


def scene(seed):
    rng = np.random.default_rng(seed)
    s = (np.arange(65) - 32) / 4.0
    psf = cpb.ImagePSF(profile(s[:, None] * s[:, None] + s[None, :] * s[None, :]), oversampling=4, normalize=False)
    y, x = 1 + (NY - 1) * rng.random(N), 1 + (NX - 1) * rng.random(N)
    u = 0.001 + rng.random(N)
    f = 100.0 / (u * u)
    f[rng.random(N) < 0.4] = 0.0
    gy, gx = np.arange(1.0, NY + 1)[:, None], np.arange(1.0, NX + 1)[None, :]
    img = np.full((NY, NX), 100.0)
    for a, b, c in zip(y, x, f):
        img = img + c * profile((gy - a) * (gy - a) + (gx - b) * (gx - b))
    iv = 1.0 / (img + 25.0)
    img = img - 100.0 + (rng.integers(0, 41, (NY, NX)) - 20)
    init = dict(y=y + 0.4 * (rng.random(N) - 0.5), x=x + 0.4 * (rng.random(N) - 0.5),
                flux=np.where(f > 0, 0.95 * f, 50.0))
    return psf, img, iv, init


def fit(seed):
    psf, img, iv, init = scene(seed)
    return cpb.fit_all_stars(img, psf, init, 6.0, n_passes=3, fixed={"bkg": 0.0}, inv_var=iv)


# nan: no quotient (flux not positive)
nan = float("nan")
EXPECTED = {
    (668, "flux"): [
        -19.44153473945756, 278.1525823422079, 209.10197533532116, 66.2823544326634, 790.1581789782405,
        378.05507364548055, 53.68086173349332, 4267.5722787166305, 21954.759015042575, 11647.673260335549,
        256.97667971478455, 55.737629586796515, -58.450201187022486, 97.41817746840728, -121.81677723771416,
        219.25218579054115, 442.0915667579516, 49.2387033699063, 66.48070543106617, 92.9409706394189,
        119.33503201815184, 3319.4150578805607, 48.2575924979936, 324.7928478998177, -48.13427593644593,
        3818.056613469027, 36.347034198720074, 4946.09369320034, 1397.6302191604143, 76.28742990199467,
        223.36386991657272, 228.6709871073779, 192.87254871464359, 76.07146351583195, 79.89306827116661,
        73.18683415904141, -36.446636663761055, 160.6911002849769, -48.046343538456426, 78.25065438176604,
    ],
    (668, "qfit"): [
        nan, 6.634626714454744, 8.230762615140137, 17.614343439969428, 1.6879806020851176, 3.0901285427841287,
        32.064182833685685, 0.3115382696280644, 0.06303531564539577, 0.14194814942834166, 5.522588373847559,
        28.429816043268357, nan, 18.20844634838004, nan, 8.835246688811687, 4.535670927077061, 39.83693706123271,
        14.553901694212275, 20.01711053571301, 12.443787692440662, 0.29475478503297137, 39.57117795859046,
        5.6699326006252155, nan, 0.5187811395886511, 42.31501251948764, 0.3111765770810979, 1.0131743311610022,
        14.85588664151713, 7.555723711785619, 7.636229187593487, 9.832058224396254, 25.96143594886179,
        23.86899731215202, 25.014034634739843, nan, 11.806084012335122, nan, 22.79833139826953,
    ],
    (505, "qfit"): [
        15.613637995923328, 32.393415350853886, 8.85540427171003, nan, 0.5799119341038519, 1.881185341039631,
        0.003773175859055445, nan, nan, 27.166944592984226, 28.841333302608053, 0.3702281907453701,
        23.741831794480674, 0.21812737184556644, 11.483694652553464, 0.02246364427296154, 11.333192142917573,
        0.27884657841712573, 11.48354094578175, nan, 6.052721232693237, 49.27342672822377, 19.52254526770915,
        6.183118754461588, 0.085455559009406, 6.026698117587857, 15.208711728113789, 5.51473830529933, nan,
        9.808068778952604, 8.67421941223991, 4.610039382530222, 0.5620790766133499, 11.669055728374822,
        10.899614797330532, 0.8821828346358874, 11.813352237888633, 3.357939616879308, nan, 0.25113426663816196,
    ],
}


@pytest.mark.parametrize("seed,key", list(EXPECTED))
def test_values_of_the_chain(seed, key):
    got, want = getattr(fit(seed), key), np.array(EXPECTED[seed, key])
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert np.linalg.norm(got[ok] - want[ok]) <= 1e-9 * np.linalg.norm(want[ok])
