"""The FP32 kernel of normal triplets holds two pixels per warp: a pixel's result must
not depend on which slot it is in, on what the other slot holds or on how many pixels
the call has.

Every pixel of a call equals, bit for bit, the same pixel inverted alone (then it is
the only one of its warp and of its launch), for counts around a warp's two slots, a
block's warps and a launch's blocks, the narrowest and widest grids, each number of
free parameters, with pixels among them that end at once (no degrees of freedom: every
sample a ghost) and steps solved by eigen-decomposition.
"""
import numpy as np
import pytest
import torch

import pmilos_b200 as pm
from gpu_common import NOISE64
from pmilos_b200 import workloads

pytestmark = pytest.mark.gpu

KEYS = ("models", "chisq", "iters", "spectra", "status")


def _cube(nl, nterms, npix):
    w = workloads.config(2 if nterms >= 10 else 1, npix=npix)
    offs = (np.arange(nl) - nl // 2) * 45.0
    w.offs, w.lam = offs, w.line.lambda0 + offs / 1000.0
    w.psf = pm.psf_gaussian(60.0, w.lam)
    w.nterms, w.miter = nterms, 12
    if nterms == 11:
        w.fix, w.guess[9] = [1] * 11, 1.0
    obs = workloads.synthesize(w, rng=np.random.default_rng(nl + npix))
    return w, obs


def _inverter(w, solver=pm.SOLVE_DEFAULT):
    return pm.Inverter(w.line, w.lam, w.psf, noise=NOISE64, fix=w.fix, nterms=w.nterms, miter=w.miter, solver=solver)


@pytest.mark.parametrize("npix", [1, 2, 3, 7, 9, 300])
@pytest.mark.parametrize("nl,nterms", [(2, 9), (5, 9), (29, 10), (3, 11), (31, 11), (32, 11), (32, 9)])
def test_a_pixel_alone_equals_the_pixel_in_a_call(nl, nterms, npix):
    w, obs = _cube(nl, nterms, npix)
    if npix > 2:
        obs[1] = -2.0  # ghosts alone: lm_mils returns before its loop
    for solver in (pm.SOLVE_DEFAULT, pm.SOLVE_EIGEN):
        if solver == pm.SOLVE_EIGEN and npix > 9:
            continue
        with _inverter(w, solver) as inv:
            x = torch.as_tensor(obs, device="cuda")
            sl = None if w.slight is None else torch.as_tensor(np.asarray(w.slight, dtype=np.float32), device="cuda")
            r = inv.invert(x, w.guess, slight=sl)
            for p in {0, 1 % npix, npix // 2, npix - 1}:
                one = inv.invert(x[p:p + 1].contiguous(), w.guess, slight=sl)
                for k in KEYS:
                    assert torch.equal(one[k][0], r[k][p]), (k, p)


def test_more_pixels_than_the_launch_has_slots():
    """Every pixel of a call that refills each slot, against the same pixels in calls
    that give each a warp of its own."""
    w, obs = _cube(15, 9, 9001)
    with _inverter(w) as inv:
        x = torch.as_tensor(obs, device="cuda")
        r = inv.invert(x, w.guess)
        assert inv.stats()["pixels"] == 9001
        for a in range(0, 9001, 1500):
            part = inv.invert(x[a:a + 1500].contiguous(), w.guess)
            for k in KEYS:
                assert torch.equal(part[k], r[k][a:a + 1500]), (k, a)
