"""The autotuner tries every launch that differs once, and none twice under two names:
what it picks among equals would be noise.  One-warp grids differ in the warps per
block (1, 2 or 4) and the staging depth alone, in both precisions; wide grids have one
launch, so their tuning stays as it was."""
import numpy as np
import pytest

import pmilos_b200 as pm
from gpu_common import case, inverter
from pmilos_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [pm.PREC_FP32, pm.PREC_FP64])
def test_one_warp_grids(precision):
    c = case(1)
    with inverter(c, precision) as inv:
        t = inv.autotune(np.tile(c["obs"], (8, 1, 1)), c["guess"], reps=1)
        assert t == inv.tuning
        assert t["variant"] == 1 and t["warps_per_block"] in (1, 2, 4) and t["staging_depth"] in (0, 2, 4)


@pytest.mark.parametrize("tuning", [(0, 2), (1, 4), (2, 4)])
def test_wide_grids(tuning):
    w = workloads.config(4, npix=16)
    obs = workloads.synthesize(w, rng=np.random.default_rng(3))
    with pm.Inverter(w.line, w.lam, w.psf, noise=w.noise, fix=w.fix) as inv:
        inv.tuning = {"variant": tuning[0], "warps_per_block": tuning[1]}
        t = inv.autotune(obs, w.guess, reps=1)
        assert (t["variant"], t["warps_per_block"], t["staging_depth"]) == (*tuning, 0)
        assert t == inv.tuning
