"""Multiplet kernels give the results they gave before triplets were sped up: models,
chi^2 and iteration counts of FP32 inversions, bit for bit.  An iteration that ends on
its data's noise floor turns a last bit into another iteration count, so a compiler
that fuses other products shows here.

The inputs and results are recorded in the golden files (Fe I 6301.5, 5P2.0-5D2.0,
profiles of drawn atmospheres with noise of 1e-3; nvcc 12.9, sm_100a)."""
import os

import numpy as np
import pytest
import torch

import pmilos_b200 as pm
from conftest import GOLDEN
from gpu_common import NOISE64

pytestmark = pytest.mark.gpu

LINE = (6301.5012, (2.0, 1.0, 2.0, 2.0, 2.0, 2.0))


def _case(file, name):
    z = np.load(os.path.join(GOLDEN, file))
    d = {k.split(".", 1)[1]: z[k] for k in z.files if k.startswith(name + ".")}
    want = {k[4:]: v for k, v in d.items() if k.startswith("out_")}
    return d, want


def _inverter(d, precision=pm.PREC_FP32):
    return pm.Inverter(pm.LineData(*LINE), d["lam"], d.get("psf"), noise=NOISE64, fix=list(d["fix"]),
                       nterms=int(9 + d["fix"][9] + d["fix"][10]), miter=30, precision=precision)


def _inverted_as_recorded(file, name):
    d, want = _case(file, name)
    dev = lambda k: None if k not in d else torch.as_tensor(d[k], device="cuda")
    with _inverter(d) as inv:
        if "lam_pix" in d:
            r = inv.invert(dev("obs"), d["guess"], slight=dev("slight"), lam=dev("lam_pix"), want_spectra=False)
            r = {k: v.cpu().numpy() for k, v in r.items()}
        else:
            r = inv.invert(d["obs"], d["guess"], slight=d.get("slight"), want_spectra=False)
    for k in want:
        assert np.array_equal(r[k], want[k]), k


@pytest.mark.parametrize("name", ["nine_33", "stray_97", "stray_97_grids", "stray_64_grids"])
def test_wide_grids(name):
    _inverted_as_recorded("wide_multiplet_results.npz", name)


@pytest.mark.parametrize("name", ["mac_15", "mac_30_grids"])
def test_one_warp_grids_with_a_v_mac_row(name):
    _inverted_as_recorded("multiplet_results.npz", name)


def test_served_grids_with_a_v_mac_row():
    """The persistent kernel's instance for several grids."""
    cases = [_case("multiplet_results.npz", f"served_{i}") for i in range(2)]
    grids = [pm.Grid(lam=d["lam"], psf=d["psf"], guess=d["guess"], noise=NOISE64, fix=list(d["fix"]), nterms=11,
                     miter=30) for d, _ in cases]
    with pm.Server(pm.LineData(*LINE), grids, hbm_budget_bytes=1 << 26) as srv:
        for i, (d, _) in enumerate(cases):
            srv.set_slight(i, d["slight"])
        ids = [srv.submit(i, d["obs"]) for i, (d, _) in enumerate(cases)]
        for (_, want), sid in zip(cases, ids):
            r = srv.wait(sid)
            for k in want:
                assert np.array_equal(r[k], want[k]), k


@pytest.mark.parametrize("name", ["synth64_10a", "synth64_10m", "synth64_11"])
def test_fp64_synthesis(name):
    """Profiles and response functions with stray light or a v_mac row."""
    d, want = _case("multiplet_results.npz", name)
    with _inverter(d, pm.PREC_FP64) as inv:
        spectra, rf = inv.synth(d["models"], rf=True, slight=d.get("slight"))
    assert np.array_equal(spectra, want["spectra"])
    assert np.array_equal(rf, want["rf"])
