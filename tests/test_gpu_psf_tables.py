"""Device tables of a PSF: only the copies that something reads.

A gridded PSF is read through its samples and their polyphase regrouping, each in Float64 and
Float32: 24 bytes a sample.  The edge-padded and the row-phase copies belong to single nodes;
a node too large for shared memory has no row-phase copies, and fits it all the same.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.photometry import Context
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu


def device_bytes(make):
    import torch
    ctx = Context(0)
    ctx.psf_handle(table_psf((33, 33), (4, 4), 1))   # the pool's first block
    free = torch.cuda.mem_get_info()[0]
    keep = [make(k) for k in range(8)]
    for p in keep:
        ctx.psf_handle(p)
    used = (free - torch.cuda.mem_get_info()[0]) / 8
    ctx.close()
    return used


def test_gridded_tables_hold_four_copies():
    nodes = [table_psf((121, 121), (4, 4), k) for k in range(16)]
    g = [1.0, 200.0, 400.0, 600.0]
    used = device_bytes(lambda k: cpb.GriddedPSFModel(nodes, [y for y in g for _ in g], [x for _ in g for x in g]))
    # 16 nodes of 121^2 samples, a polyphase copy of at most 31^2 * 16 each; blocks come in 2 MB
    assert used <= 16 * (12 * 121 ** 2 + 12 * 124 ** 2) + (4 << 20)


@pytest.mark.parametrize("size", [(101, 101), (161, 157), (221, 217), (401, 397)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nodes_on_either_side_of_shared_memory(size, precision):
    """All row-phase copies; all but fit_star's; the Float32 one; none.  Tolerances: test_gpu_stamp_kernel's."""
    from oracle import orc_fit_simultaneous
    psf, rng = table_psf(size, (4, 4), 5), np.random.default_rng(size[0])
    img, iv = rng.normal(10.0, 1.0, (61, 57)), rng.uniform(0.5, 2.0, (61, 57))
    src = dict(y=np.array([16.3, 44.8]), x=np.array([18.6, 37.1]), flux=np.array([500.0, 700.0]))
    kw = dict(fixed={"bkg": 0.0}, inv_var=iv, model_rad=9, max_iter=2 if precision == "fp64" else 1)
    g = cpb.fit_all_stars_simultaneous(img, psf, src, 7, precision=precision, **kw)
    o = orc_fit_simultaneous(img, psf, src, 7, **kw)
    tol = 1e-9 if precision == "fp64" else 3e-5
    for k in ("y", "x", "flux"):
        np.testing.assert_allclose(getattr(g, k), getattr(o, k), rtol=tol, atol=tol)
    m = cpb.fit_all_stars(img - 10.0, psf, src, 7, n_passes=1, fixed={"bkg": 0.0}, inv_var=iv, max_iter=1)
    assert np.isfinite(m.residual).all()
