"""Fits with small and large tables on two contexts at once.

A kernel's limit of dynamic shared memory belongs to the kernel on its device: a thread that
fits with a small table must not lower it between another thread's setting it and launching
with a large one (that launch is refused).  Two threads with a context each run the same
kernels over tables, boxes and groups of different sizes; every call succeeds and has the
bits of the same call alone.
"""
import threading

import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.photometry import Context
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu
KEYS = ("y", "x", "flux", "chisq", "qfit", "spread_model")


def calls(size, R, seed):
    """The fitters over a table of `size` samples and boxes of radius R, each as a function of a context."""
    rng = np.random.default_rng(seed)
    psf, shape, n = table_psf(size, (4, 4), seed), (150, 141), 60
    img, iv = rng.normal(0, 3, shape), np.full(shape, 0.1)
    g = 12.0 + 16.0 * np.stack(np.meshgrid(np.arange(8), np.arange(8), indexing="ij"))
    src = dict(y=g[0].ravel()[:n] + rng.uniform(-1, 1, n), x=g[1].ravel()[:n] + rng.uniform(-1, 1, n),
               flux=rng.uniform(500, 1500, n))
    kw = dict(fixed={"bkg": 0.0}, inv_var=iv, max_iter=2)
    k = 4                      # groups: stars on a diagonal of one small image
    side = 2 * R + 4 * k
    pix = rng.normal(0, 3, side * side)
    at = R + 1 + 3.5 * np.arange(k)

    def star(ctx):
        b, r = cpb.fit_star(cpb.replace_params(psf, y=30.2, x=28.8, flux=900.0), img, ((30 - R, 30 + R), (29 - R, 29 + R)),
                            fixed={"bkg": 0.0}, inv_var=iv, ctx=ctx)
        return dict(y=np.array(b.y), x=np.array(b.x), flux=np.array(b.flux), chisq=np.array(r.chisq))

    def groups(ctx):
        return cpb.fit_groups_packed(psf, pix, [0], [side], [side], [0, k], at, at + 0.3, np.full(k, 900.0), R,
                                     inv_var=np.full(side * side, 0.1), fixed={"bkg": 0.0}, model_rad=R, max_iter=2,
                                     ctx=ctx)

    return [lambda ctx: vars(cpb.fit_all_stars_simultaneous(img, psf, src, float(R), model_rad=float(R), ctx=ctx, **kw)),
            lambda ctx: vars(cpb.fit_all_stars_simultaneous(img, psf, src, float(R), model_rad=float(R), ctx=ctx,
                                                            precision="mixed", **kw)),
            lambda ctx: vars(cpb.fit_all_stars(img, psf, src, float(R), n_passes=1, ctx=ctx, **kw)), star, groups]


def test_small_and_large_tables_side_by_side():
    sides = [calls((17, 17), 3, 1), calls((101, 101), 12, 2)]
    want = []
    for side in sides:
        ctx = Context(0)
        want.append([c(ctx) for c in side])
        ctx.close()
    errors, start = [], threading.Barrier(2)

    def work(k):
        try:
            ctx = Context(0)
            start.wait()
            for _ in range(25):
                for c, w in zip(sides[k], want[k]):
                    r = c(ctx)
                    for q in KEYS:
                        assert q not in w or np.array_equal(r[q], w[q], equal_nan=True), q
            ctx.close()
        except BaseException as e:
            errors.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not errors, errors
