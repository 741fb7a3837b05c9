"""The FP32 kernel of normal triplets where a pixel ends at once (as many degrees of
freedom as parameters: lm_mils returns before its loop, milosUtils.c:507-512), in
either slot of a warp, next to pixels that go on, in runs and in whole calls; and the
same bits from every launch shape that the kernel has.
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
    w.offs = (np.arange(nl) - nl // 2) * 45.0
    w.lam = w.line.lambda0 + w.offs / 1000.0
    w.psf = pm.psf_gaussian(60.0, w.lam)
    w.nterms, w.miter = nterms, 12
    if nterms == 11:
        w.fix, w.guess[9] = [1] * 11, 1.0
    return w, workloads.synthesize(w, rng=np.random.default_rng(nl + npix))


def _inverter(w):
    return pm.Inverter(w.line, w.lam, w.psf, noise=NOISE64, fix=w.fix, nterms=w.nterms, miter=w.miter,
                       classical=False)


def _slight(w):
    return None if w.slight is None else np.asarray(w.slight, dtype=np.float32)


def _on_device(inv, w, obs):
    sl = _slight(w)
    r = inv.invert(torch.as_tensor(obs, device="cuda"), w.guess,
                   slight=None if sl is None else torch.as_tensor(sl, device="cuda"))
    return {k: v.cpu().numpy() for k, v in r.items()}


def _end_at_once(obs, which, nterms):
    """Exactly nterms samples of these pixels are left, the rest ghosts: nfree = 0."""
    out = obs.copy()
    out.reshape(obs.shape[0], -1)[which, nterms:] = -2.0
    return out


# which pixels end at once
PATTERNS = {"first": lambda n: [0], "last": lambda n: [n - 1], "odd": lambda n: list(range(1, n, 2)),
            "run": lambda n: list(range(n // 4, n - n // 4)), "all": lambda n: list(range(n))}


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("npix", [2, 9, 1500, 6001])
@pytest.mark.parametrize("nl,nterms", [(4, 9), (15, 10), (32, 11)])
def test_pixels_that_end_at_once(nl, nterms, npix, pattern):
    w, obs = _cube(nl, nterms, npix)
    ended = np.zeros(npix, dtype=bool)
    ended[PATTERNS[pattern](npix)] = True
    masked = _end_at_once(obs, ended, nterms)
    with _inverter(w) as inv:
        whole = _on_device(inv, w, obs)
        # the device call and, by its size, the replayed graph or the fed call
        for r in (_on_device(inv, w, masked), inv.invert(masked, w.guess, slight=_slight(w))):
            assert np.all(r["status"][ended] == pm.PIX_NFREE) and np.all(r["iters"][ended] == -1)
            assert np.all(r["chisq"][ended] == 0) and np.all(r["spectra"][ended] == 0)
            assert np.all(r["models"][ended] == np.asarray(w.guess))
            for k in KEYS:
                assert np.array_equal(r[k][~ended], whole[k][~ended]), k


def test_served_scans_of_pixels_that_end_at_once():
    """Scans on two grids of which one ends whole and one in part, among others."""
    ws = [_cube(nl, 9, 700) for nl in (6, 30)]
    grids = [pm.Grid(lam=w.lam, psf=w.psf, guess=w.guess, noise=NOISE64, fix=w.fix, nterms=9, miter=w.miter,
                     classical=False) for w, _ in ws]
    odd = np.arange(700) % 2 == 1
    scans = [(0, ws[0][1]), (1, _end_at_once(ws[1][1], np.ones(700, dtype=bool), 9)), (1, ws[1][1]),
             (0, _end_at_once(ws[0][1], odd, 9)), (1, _end_at_once(ws[1][1], odd, 9))]
    with pm.Server(ws[0][0].line, grids, hbm_budget_bytes=1 << 26) as srv:
        r = [srv.wait(i) for i in [srv.submit(g, x) for g, x in scans]]
    assert np.all(r[1]["status"] == pm.PIX_NFREE) and np.all(r[1]["iters"] == -1)
    for part, full in ((3, 0), (4, 2)):
        assert np.all(r[part]["status"][odd] == pm.PIX_NFREE)
        for k in ("models", "chisq", "iters", "status"):
            assert np.array_equal(r[part][k][~odd], r[full][k][~odd]), k


@pytest.mark.parametrize("npix", [1500, 3000])  # a warp per pixel, and more pixels than warps
@pytest.mark.parametrize("nterms", [9, 10])
def test_every_launch_shape_gives_the_same_bits(nterms, npix):
    """Each variant and block size, with the pixel count published before the launch
    (device) and while the kernel runs (host, whole or in pieces)."""
    w, obs = _cube(30, nterms, npix)
    with _inverter(w) as inv:
        ref = _on_device(inv, w, obs)
        for variant, wpb in ((0, 1), (0, 4), (1, 2), (2, 4), (2, 16)):
            inv.tuning = {"variant": variant, "warps_per_block": wpb, "staging_depth": 0}
            rs = [_on_device(inv, w, obs), inv.invert(obs, w.guess, slight=_slight(w))]
            inv.tuning = {"staging_depth": 3}
            rs.append(inv.invert(obs, w.guess, slight=_slight(w)))
            for r in rs:
                for k in KEYS:
                    assert np.array_equal(r[k], ref[k]), (k, variant, wpb)
