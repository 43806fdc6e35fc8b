"""fit_star batches over the forms of the batched kernel, against the oracle's fit_star.

One warp and four warps a cutout (large and small batches); nodes that fit shared memory
and nodes that do not (read from the padded polyphase copy); free sets that are and are
not the leading parameters, of every count; cutouts staged in shared memory and cutouts
too large for it, 1-pixel-wide ones, with and without weights, both pixel types; stars at
whole pixels whose stencils hit the first and the last table sample.  Tolerance: the
normal matrices of these fits have condition numbers below 1e5 after scaling, so FP64
rounding stays below 1e-10 relative; 1e-8 is asked for, as of the other batched fits.
"""
import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200 import GriddedPSFModel
from crowdphot_b200.simulate import psf_value
from test_gpu_stamp_kernel import table_psf

pytestmark = pytest.mark.gpu
NAMES = ("y", "x", "flux", "bkg")


@pytest.mark.parametrize("size,os_,fixed,n,dtype,weights", [
    ((33, 33), (4, 4), {"bkg": 0.0}, 7, np.float64, True),       # staged node, leading free set, 4 warps
    ((33, 33), (4, 4), {"bkg": 0.0}, 640, np.float32, True),     # one warp
    ((33, 33), (4, 4), {}, 9, np.float32, False),
    ((25, 31), (3, 2), {"flux": 5000.0}, 8, np.float64, True),   # y, x, bkg: not the leading three
    ((25, 31), (1, 5), {"y": 0.0, "x": 0.0}, 6, np.float64, True),
    ((33, 33), (4, 4), {"y": 0.0, "x": 0.0, "bkg": 0.0}, 5, np.float64, False),
    ((181, 181), (4, 4), {"bkg": 0.0}, 7, np.float64, True),     # 262 KB node: not staged
    ((181, 181), (4, 4), {}, 640, np.float32, True),
    ((181, 181), (4, 4), {"x": 0.0, "bkg": 0.0}, 6, np.float64, True),
])
def test_batches_match_the_oracle(size, os_, fixed, n, dtype, weights):
    from oracle import orc_fit_star
    psf = table_psf(size, os_, seed=size[0] + n)
    node = GriddedPSFModel([psf], [0.0], [0.0])
    rng = np.random.default_rng(n + size[1])
    imgs, ivs, org, inits = [], [], [], []
    for i in range(n):
        h, w = (7, 7) if i % 4 == 0 else (int(rng.integers(6, 15)), int(rng.integers(6, 15)))
        if i == 1:
            h, w = 61, 67   # beyond the staged size of a team
        if i == 2:
            h, w = 15, 1
        y1, x1 = int(rng.integers(1, 30)), int(rng.integers(1, 30))
        yc, xc = y1 + (h - 1) / 2, x1 + (w - 1) / 2
        if i % 4:   # every fourth star starts and lies at a whole pixel
            yc, xc = yc + rng.uniform(-0.4, 0.4), xc + rng.uniform(-0.4, 0.4)
        yy, xx = np.meshgrid(np.arange(y1, y1 + h, dtype=float), np.arange(x1, x1 + w, dtype=float), indexing="ij")
        img = psf_value(node, yc, xc, 5000.0, yy, xx) + rng.normal(0, 2.0, (h, w))
        fy, fx = fixed.get("y"), fixed.get("x")
        init = np.array([yc if fy is not None else yc + rng.normal(0, 0.1) * (i % 4 > 0),
                         xc if fx is not None else xc + rng.normal(0, 0.1) * (i % 4 > 0), 4700.0, 0.5])
        for k, v in fixed.items():
            if k in ("flux", "bkg"):
                init[NAMES.index(k)] = v
        imgs.append(img.astype(dtype))
        ivs.append(rng.uniform(0.1, 0.4, (h, w)).astype(dtype))
        org.append((y1, x1))
        inits.append(init)
    if "y" in fixed or "x" in fixed:   # one value for all: the free ones then fit around it
        fixed = {k: (float(np.mean([o[0] + 3 for o in org])) if k == "y" else
                     float(np.mean([o[1] + 3 for o in org])) if k == "x" else v) for k, v in fixed.items()}
        for v in inits:
            for k in fixed:
                v[NAMES.index(k)] = fixed[k]
    out = cpb.fit_star_batch(psf, imgs, inv_vars=ivs if weights else None, origins=org, inits=inits, fixed=fixed,
                             max_iter=40)
    same = 0
    for i in range(n):
        (y1, x1), (h, w) = org[i], imgs[i].shape
        full = np.zeros((y1 + h - 1, x1 + w - 1), dtype)
        fiv = np.zeros_like(full)
        full[y1 - 1:, x1 - 1:] = imgs[i]
        fiv[y1 - 1:, x1 - 1:] = ivs[i]
        model = cpb.replace_params(psf, **dict(zip(NAMES, inits[i])))
        try:
            best, res = orc_fit_star(model, full, ((y1, y1 + h - 1), (x1, x1 + w - 1)),
                                     inv_var=fiv if weights else None, fixed=fixed, max_iter=40)
        except cpb.ArgumentError:
            assert out["status"][i] != 0
            same += 1
            continue
        assert out["status"][i] == 0
        if out["iterations"][i] != res.iterations or not res.converged or w == 1:
            same += out["iterations"][i] == res.iterations
            continue
        same += 1
        ref = np.array([getattr(best, k) for k in NAMES])
        np.testing.assert_allclose(out["params"][i], ref, rtol=1e-8, atol=1e-6)
        np.testing.assert_allclose(out["chisq"][i], res.chisq, rtol=1e-8)
    assert same >= 0.98 * n
