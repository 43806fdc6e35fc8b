"""The worker threads of large pageable copies: no more than processors, but one a context.

A context's workers are the threads that its first large fit adds to the process.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import crowdphot_b200 as cpb
from crowdphot_b200.photometry import Context

pytestmark = pytest.mark.gpu
PSF = cpb.CircularGaussianPSF(fwhm=2.5)


def fit(ctx, side, n=4):
    rng = np.random.default_rng(side)
    img, iv = rng.normal(0, 3, (side, side)), np.full((side, side), 0.1)
    src = dict(y=rng.uniform(5, side - 5, n), x=rng.uniform(5, side - 5, n), flux=rng.uniform(500, 1500, n))
    return cpb.fit_all_stars_simultaneous(img, PSF, src, 3.0, fixed={"bkg": 0.0, "fwhm": 2.5}, inv_var=iv, model_rad=3.0,
                                          max_iter=1, ctx=ctx)


def threads():
    return set(os.listdir("/proc/self/task"))


def counts(cores):
    """Threads that two contexts' first large fits add in a process that may use `cores` processors."""
    os.sched_setaffinity(0, sorted(os.sched_getaffinity(0))[:cores])
    out, held = [], []
    for _ in range(2):
        ctx = Context(0)
        held.append(ctx)
        fit(ctx, 120)
        t0 = threads()
        fit(ctx, 1100)
        out.append(len(threads() - t0))
    return out


@pytest.mark.parametrize("cores,most", [(1, [1, 1]), (2, [2, 1]), (3, [3, 1])])
def test_workers_are_bounded_by_the_processors(cores, most):
    if len(os.sched_getaffinity(0)) < cores:
        pytest.skip("fewer processors")
    code = f"import sys; sys.path[:0] = {sys.path!r}\nimport json, test_gpu_copy_workers as t; print(json.dumps(t.counts({cores})))"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=os.path.dirname(__file__))
    assert r.returncode == 0, r.stderr[-2000:]
    assert json.loads(r.stdout.strip().splitlines()[-1]) == most
