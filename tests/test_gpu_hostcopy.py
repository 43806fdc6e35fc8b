"""Large pageable copies run over worker threads; pinned and small ones through the driver.

The same fit from pageable and from pinned memory must give the same bits: inputs and the
residual image on either side of the size limit, with sizes that are no multiple of a
copy chunk, several fits on one context, and two contexts in two threads.
"""
import ctypes as C
import threading

import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200 import _abi
from crowdphot_b200.photometry import Context, SimOutputs, sim_params
from crowdphot_b200.simulate import moffat_epsf

pytestmark = pytest.mark.gpu


def field(shape, dtype, seed):
    rng = np.random.default_rng(seed)
    img = np.asfortranarray(rng.normal(50, 7, shape), dtype=dtype)
    iv = np.asfortranarray(rng.uniform(0.01, 0.03, shape), dtype=dtype)
    bkg = np.asfortranarray(rng.uniform(45, 55, shape), dtype=dtype)
    n = 20
    src = [rng.uniform(5, shape[0] - 5, n), rng.uniform(5, shape[1] - 5, n), rng.uniform(300, 900, n)]
    return img, iv, bkg, src


def fit(ctx, psf, shape, img, iv, bkg, src, pinned):
    import torch
    keep = []

    def place(a):
        if not pinned:
            return a.copy(order="F")
        t = torch.from_numpy(np.ascontiguousarray(a.T)).pin_memory()
        keep.append(t)
        return t.numpy().T

    a = [place(v) for v in (img, iv, bkg)]
    outs = SimOutputs(20, *shape, 0, residual=True)
    if pinned:
        outs.residual = place(outs.residual)
        outs.c.residual = outs.residual.ctypes.data_as(_abi._dp)
    P = sim_params(psf, 5, {"bkg": 0.0}, inv_var_given=True, model_rad=5, max_iter=3)
    vp = lambda x: x.ctypes.data_as(C.c_void_p)
    dp = lambda x: x.ctypes.data_as(_abi._dp)
    et = _abi.CPB_F32 if img.dtype == np.float32 else _abi.CPB_F64
    rc = ctx.lib.cpb_fit_simultaneous(ctx.handle, ctx.psf_handle(psf), C.byref(P), vp(a[0]), et, *shape, vp(a[1]),
                                      vp(a[2]), 20, dp(src[0]), dp(src[1]), dp(src[2]), C.byref(outs.c))
    ctx.raise_for(rc, "cpb_fit_simultaneous")
    return np.array(outs.residual), outs.y.copy(), outs.flux.copy(), outs.chisq.copy()


# below the limit; inputs just above it and the residual below; both above; many chunks
@pytest.mark.parametrize("shape,dtype", [((301, 150), np.float32), ((837, 838), np.float32), ((1031, 1021), np.float32),
                                         ((1503, 1201), np.float64)])
def test_pageable_and_pinned_fits_have_the_same_bits(shape, dtype):
    ctx, psf = Context(0), moffat_epsf()
    for seed in (1, 2, 3):
        f = field(shape, dtype, seed)
        for a, b in zip(fit(ctx, psf, shape, *f, False), fit(ctx, psf, shape, *f, True)):
            assert np.array_equal(a, b, equal_nan=True)
    ctx.close()


def test_two_contexts_in_two_threads():
    shape, psf = (1100, 1001), moffat_epsf()
    fields = [field(shape, np.float32, s) for s in (5, 6)]
    want = []
    for f in fields:
        ctx = Context(0)
        want.append(fit(ctx, psf, shape, *f, True))
        ctx.close()
    got = [[], []]

    def work(k):
        ctx = Context(0)
        for _ in range(4):
            got[k].append(fit(ctx, psf, shape, *fields[k], False))
        ctx.close()

    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    [t.start() for t in th]
    [t.join() for t in th]
    for k in (0, 1):
        assert len(got[k]) == 4
        for r in got[k]:
            assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(r, want[k]))
