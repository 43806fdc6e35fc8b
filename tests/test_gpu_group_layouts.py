"""A group's result does not depend on the launch that fits it.

Fit half-width 6, model radius 9, tabulated PSF: a 12-star group in a 39 x 45 or 41 x 41 image
fits half an SM with room for its whole image, so alone it is one launch of the full layout.
In a batch led by a 14-star group the half-SM layout runs first: 109,568 bytes an SM's half,
less 24 + 2 bytes for each of 14 * 169 stamp entries, leave room for at most 1,716 union
pixels of 28 bytes.  There the tight 12-star blend is fitted by the half launch and the group
whose boxes cover all 1,755 pixels of its image is deferred to the second one.  Same block size
in each, so the same bits.
"""
import numpy as np
import pytest

from crowdphot_b200.photometry import Context
from test_gpu_group_forms import pack
from test_gpu_groups import run_batch
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu
R, KEYS = 6, ("y", "x", "flux", "y_err", "x_err", "flux_err", "chisq", "qfit", "qfit_z", "crowding", "spread_model",
              "n_iter", "valid")


def batch(seed):
    rng = np.random.default_rng(seed)
    groups = []

    def group(ny, nx, y, x):
        jit = lambda v: np.asarray(v, float) + rng.uniform(-0.2, 0.2, len(v))
        groups.append((ny, nx, jit(y), jit(x), rng.uniform(2e3, 8e3, len(y))))

    # places within 0.3 px of integers, guesses included: those are the anchors
    g = np.arange(14)
    group(70, 61, 12 + 9 * (g // 4), 12 + 9 * (g % 4))                       # leads the half launch
    cover = np.array([7, 17, 28, 39])
    group(39, 45, np.repeat([7, 20, 33], 4), np.tile(cover, 3))              # union: the whole image
    g = np.arange(12)
    group(41, 41, 14 + 4 * (g // 4), 13 + 4 * (g % 4))                       # tight
    psf = table_psf((81, 81), (4, 4), 3)
    d = pack(psf, groups, np.float64, seed)
    d["inv_var"] = rng.uniform(0.5, 1.5, d["pix"].size)                       # every pixel usable
    return psf, d


def launches(ctx):
    return ctx.kernel_stats()[0]["k_groups"]["launches"]


@pytest.mark.parametrize("seed", [1, 2])
def test_full_half_and_deferred_give_the_same_bits(seed):
    psf, d = batch(seed)
    kw = dict(fixed={"bkg": 0.0}, model_rad=9, max_iter=12, residual=True)
    ctx = Context(0)
    ctx.set_profiling(True)
    ctx.kernel_stats()
    both = run_batch(psf, d, R, ctx=ctx, **kw)
    assert launches(ctx) == 2 and both["n_kernel_groups"] == 3
    assert both["n_union"][1] == 39 * 45 and both["n_union"][2] < 1000 and both["n_union"][0] <= 14 * 169
    for g in (1, 2):
        s0, s1, o = d["star_offsets"][g], d["star_offsets"][g + 1], d["offsets"][g]
        n = int(d["ny"][g]) * int(d["nx"][g])
        one = dict(pix=d["pix"][o:o + n], inv_var=d["inv_var"][o:o + n], offsets=np.zeros(1, np.int64),
                   ny=d["ny"][g:g + 1], nx=d["nx"][g:g + 1], star_offsets=np.array([0, s1 - s0], np.int64),
                   y=d["y"][s0:s1], x=d["x"][s0:s1], flux=d["flux"][s0:s1])
        r = run_batch(psf, one, R, ctx=ctx, **kw)
        assert launches(ctx) == 1
        for k in KEYS:
            np.testing.assert_array_equal(r[k], both[k][s0:s1], err_msg=f"{g} {k}")
        np.testing.assert_array_equal(r["residual"][:n], both["residual"][o:o + n])
    ctx.close()
