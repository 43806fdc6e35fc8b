"""Device tables live as long as something may read them, and no longer.

A loop that makes a model a star (replace_params) uploads a table each; those of models that
are gone are given back.  Tables behind a handle from psf_handle stay until the context is
closed, those of a BatchGraph as long as the graph.
"""
import ctypes as C
import gc
import threading

import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200 import _abi
from crowdphot_b200.photometry import Context, SimOutputs, _lm_outputs, sim_params
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu


def scene(seed=1, shape=(41, 39)):
    rng = np.random.default_rng(seed)
    return rng.normal(0, 3, shape), np.full(shape, 0.1)


def star(psf, ctx):
    img, iv = scene()
    return cpb.fit_star(cpb.replace_params(psf, y=20.2, x=19.1, flux=900.0), img, fixed={"bkg": 0.0}, inv_var=iv,
                        ctx=ctx)[0]


def churn(ctx, n=60):
    """Uploads and drops tables of several sizes, so that any given back early are written over."""
    for k in range(n):
        star(table_psf((33 + 4 * (k % 18), 101), (4, 4), k), ctx)


def test_memory_stays_flat_over_new_models():
    import torch
    ctx, psf = Context(0), table_psf((101, 101), (4, 4), 1)
    want = star(psf, ctx)
    free = torch.cuda.mem_get_info()[0]
    for _ in range(400):   # 0.56 MB of tables each
        b = star(psf, ctx)
        assert (b.y, b.x, b.flux) == (want.y, want.x, want.flux)
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20   # blocks of the pool
    assert len(ctx._psfs) <= 2
    ctx.close()


def test_handed_out_handles_outlive_their_model():
    ctx = Context(0)
    img, iv = (np.asfortranarray(a) for a in scene(2, (60, 50)))
    src = [np.array([20.0, 41.0]), np.array([15.0, 33.0]), np.array([800.0, 900.0])]

    def fit(hp, psf):
        outs = SimOutputs(2, 60, 50, 0, residual=True)
        P = sim_params(psf, 6, {"bkg": 0.0}, inv_var_given=True, model_rad=6, max_iter=3)
        vp, dp = lambda a: a.ctypes.data_as(C.c_void_p), lambda a: a.ctypes.data_as(_abi._dp)
        ctx.raise_for(ctx.lib.cpb_fit_simultaneous(ctx.handle, hp, C.byref(P), vp(img), _abi.CPB_F64, 60, 50, vp(iv), None,
                                                   2, *map(dp, src), C.byref(outs.c)), "fit")
        return np.array(outs.residual)

    psf = table_psf((101, 101), (4, 4), 7)
    hp = ctx.psf_handle(psf)
    want = fit(hp, psf)
    like = table_psf((33, 33), (4, 4), 7)   # any ImagePSF: the parameters do not name the table
    del psf
    gc.collect()
    churn(ctx)
    assert np.array_equal(fit(hp, like), want)
    ctx.close()


def test_a_graph_keeps_its_tables():
    import torch
    ctx, n = Context(0), 5
    img, iv = scene(3, (25, 25))
    cuda = lambda a, d: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device="cuda")
    lm = dict(offsets=cuda(np.arange(n) * 625, torch.int64), ny=cuda(np.full(n, 25), torch.int32),
              nx=cuda(np.full(n, 25), torch.int32), y1=cuda(np.ones(n), torch.int32), x1=cuda(np.ones(n), torch.int32),
              pix=cuda(np.tile(img.ravel(), n), torch.float64), inv_var=cuda(np.tile(iv.ravel(), n), torch.float64),
              init=cuda([[12.5 + 0.1 * k, 13.0, 900.0, 0.0] for k in range(n)], torch.float64),
              out={k: torch.from_numpy(v).cuda() for k, v in _lm_outputs(n, 4, 3).items()})
    graph = cpb.BatchGraph(table_psf((101, 101), (4, 4), 9), lm=lm, lm_fixed={"bkg": 0.0}, autotune=0, ctx=ctx)
    graph.launch()
    want = lm["out"]["params"].cpu().numpy()
    gc.collect()
    churn(ctx)
    lm["out"]["params"].zero_()
    graph.launch()
    assert np.array_equal(lm["out"]["params"].cpu().numpy(), want)
    graph.close()
    ctx.close()


def test_threads_share_a_context():
    ctx, psfs = Context(0), [table_psf((65 + 4 * k, 61), (4, 4), k) for k in range(3)]
    want = [star(p, ctx) for p in psfs]
    errors = []

    def work(k):
        try:
            for _ in range(60):
                b = star(psfs[k], ctx)
                assert (b.y, b.x, b.flux) == (want[k].y, want[k].x, want[k].flux)
        except BaseException as e:
            errors.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not errors, errors
    ctx.close()
