"""Simultaneous fits of more than one star on 32 pixels.

There the J^T u kernel has more blocks than any kernel over the pixels or the parameters, and
every block's partial sum needs its place.  Against the oracle after one outer iteration (a
few inner ones: such a field is ill-conditioned, so rounding grows with each), and bit for bit
between a context alone and two contexts working side by side.
"""
import threading

import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.photometry import Context
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu
KEYS = ("y", "x", "flux", "chisq", "qfit")


def field(shape, n, seed):
    rng = np.random.default_rng(seed)
    psf = table_psf((33, 33), (4, 4), 2)
    img, iv = rng.normal(20, 3, shape), np.full(shape, 0.1)
    src = dict(y=rng.uniform(2, shape[0] - 1, n), x=rng.uniform(2, shape[1] - 1, n), flux=rng.uniform(300, 900, n))
    return (img, psf, src, 4.0), dict(fixed={"bkg": 0.0}, inv_var=iv, model_rad=4.0)


@pytest.mark.parametrize("shape,n", [((60, 61), 300), ((100, 97), 900), ((33, 40), 640)])
def test_one_iteration_matches_the_oracle(shape, n):
    from oracle import orc_fit_simultaneous
    args, kw = field(shape, n, n)
    kw.update(max_iter=1, inner_iterations=3)
    g, o = cpb.fit_all_stars_simultaneous(*args, **kw), orc_fit_simultaneous(*args, **kw)
    for k in ("y", "x", "flux", "residual"):
        np.testing.assert_allclose(getattr(g, k), getattr(o, k), rtol=1e-7, atol=1e-7)


def test_two_contexts_side_by_side_give_the_same_bits():
    calls = []
    for shape, n in (((100, 97), 900), ((64, 60), 500)):
        args, kw = field(shape, n, n + 1)
        kw.update(max_iter=4)
        calls.append(lambda ctx, a=args, k=kw: cpb.fit_all_stars_simultaneous(*a, ctx=ctx, **k))
    want = []
    for call in calls:
        ctx = Context(0)
        want.append(call(ctx))
        ctx.close()
    errors, start = [], threading.Barrier(2)

    def work(k):
        try:
            ctx = Context(0)
            calls[k](ctx)
            start.wait()
            for _ in range(60):
                r = calls[k](ctx)
                for q in KEYS:
                    assert np.array_equal(getattr(r, q), getattr(want[k], q), equal_nan=True)
            ctx.close()
        except BaseException as e:
            errors.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not errors, errors
