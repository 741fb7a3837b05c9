"""A resident server whose scans come slowly: most warps of the persistent kernel hold
tickets that a trickle of small scans does not reach for minutes, and must not take
that for a stalled queue.

The kernel gives up 30 s + max(1 s, 2 linger) after the last sign of its producer: 32 s
with a linger of 1 s.  Scans of 8 pixels every half second keep it running (each pause
is shorter than the linger) for longer than that."""
import time

import numpy as np
import pytest

import pmilos_b200 as pm
from gpu_common import NOISE64
from pmilos_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [pm.PREC_FP32, pm.PREC_FP64], ids=["two-pixel kernel", "one-pixel kernel"])
def test_small_scans_for_longer_than_the_wait_limit(precision):
    w = workloads.config(1, npix=8)
    obs = workloads.synthesize(w, rng=np.random.default_rng(5))
    grid = pm.Grid(lam=w.lam, psf=w.psf, guess=w.guess, noise=NOISE64, fix=w.fix, nterms=9, precision=precision)
    with pm.Server(w.line, [grid], hbm_budget_bytes=1 << 24, linger_ms=1000.0) as srv:
        first = srv.wait(srv.submit(0, obs))
        end = time.monotonic() + 34.0
        while time.monotonic() < end:
            time.sleep(0.5)
            r = srv.wait(srv.submit(0, obs))
        assert np.array_equal(r["models"], first["models"])
        assert srv.stats()["kernel_launches"] == 1  # the kernel ran all the while
