"""What is measured: the calls a user of the package makes, from one pixel of a
host's own loop to whole cubes, over the wavelength grids, stray-light modes,
precisions and memories that the package takes.

Every inversion's input is a cube of synthetic observed profiles: atmospheres
drawn from the package's own workload distributions, synthesized here in plain
64-bit torch (the Milne-Eddington solution with the Hui et al. 1978 Voigt
function), correlated with the instrumental profile, plus Gaussian noise of 1e-3
of the continuum.  Inputs depend on the seed alone.

A case is a dict:
  kind      lm_mils | host | pinned | device | synth | server | fits
  npix      pixels (server: of each scan)
  nl        wavelengths
  fwhm      width of the instrumental profile [mA], 0 for none
  slight    none | shared | pixel: stray light (with the filling factor as a tenth parameter)
  mac       macroturbulence as an eleventh parameter
  line      triplet (Fe I 6173, 5P1.0-5D0.0) or multiplet (Fe I 6301.5, 5P2.0-5D2.0)
  precision fp32 (the default form) | fp64 (the plain form)
  scans     server: scans per pass
  order     fits: axis roles of NAXIS1..4 (L wavelength, S Stokes, R rows, C columns)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "p-milos_b200"))

import pmilos_b200 as pm  # noqa: E402
from pmilos_b200 import specs  # noqa: E402

# LM steps and accepted steps of a pixel of the ordinary cube (30 wavelengths, nine
# parameters): the path's work follows the data, these are its means
STEPS, ACCEPTED = 29, 15
SERVER_GRIDS = (6, 15, 30)
NOISE = (1.0 / specs.SN) ** 2
LINES = {"triplet": (specs.FE6173, specs.TRIPLET), "multiplet": (6301.5012, (2.0, 1.0, 2.0, 2.0, 2.0, 2.0))}
BASE = {"nl": 30, "fwhm": 60.0, "slight": "none", "mac": False, "line": "triplet", "precision": "fp32"}


def listed():
    def case(name, kind, npix, **more):
        return {"name": name, "kind": kind, "npix": npix, **BASE, **more}

    return [
        # a host that keeps its per-pixel loop: one lm_mils call at a time
        case("pixel_lm_mils", "lm_mils", 1),
        # one slit position of a raster scan, from and to ordinary host arrays
        case("slit_host", "host", 512),
        # the ordinary cube, already on the GPU (256 x 256 pixels)
        case("cube_device", "device", 65536),
        # the same from pinned host arrays to pinned host arrays, as a scan loop holds them
        case("cube_pinned", "pinned", 83333),
        # a larger cube with stray light: a shared profile and the filling factor inverted
        case("stray_light_device", "device", 262144, slight="shared"),
        # a filtergraph's 15 positions
        case("grid15_device", "device", 65025, nl=15),
        # a spectrograph's 112 points
        case("wide112_device", "device", 65536, nl=112, fwhm=25.0),
        # the plain form on a small cube without an instrumental profile: the check of a set-up
        case("plain_fp64", "device", 4096, fwhm=0.0, precision="fp64"),
        # macroturbulence inverted as well (eleven parameters)
        case("macroturbulence", "device", 16384, slight="shared", mac=True),
        # forward synthesis with response functions of a cube of models
        case("synth_rf", "synth", 65536),
        # a real-time loop: scans on three grids through the resident server
        case("server_scans", "server", 10000, nl=30, scans=9),
        # a cube file in the reference's default axis order
        case("ingest_fits", "fits", 256 * 250, order="LSRC"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    c = dict(BASE)
    kind = rng.choice(["device", "device", "device", "wide", "wide", "host", "pinned", "synth", "fits", "mac", "fp64",
                       "lm_mils", "server"])
    c["nl"] = rng.randint(6, 32)
    c["fwhm"] = rng.choice([0.0, round(rng.uniform(30.0, 90.0), 1), round(rng.uniform(30.0, 90.0), 1)])
    c["kind"] = kind if kind not in ("wide", "mac", "fp64") else "device"
    if kind == "device":
        c["npix"] = _log(rng, 300, 100000)
        c["slight"] = rng.choice(["none", "none", "shared", "pixel"])
        c["line"] = rng.choice(["triplet", "triplet", "triplet", "multiplet"])
    elif kind == "wide":
        c["npix"] = _log(rng, 200, 30000)
        c["nl"] = rng.randint(33, 120)
        c["fwhm"] = rng.choice([0.0, round(rng.uniform(15.0, 40.0), 1)])
        c["slight"] = rng.choice(["none", "none", "shared"])
    elif kind == "host":
        c["npix"] = _log(rng, 2, 20000)
        c["slight"] = rng.choice(["none", "none", "pixel"])
    elif kind == "pinned":
        c["npix"] = _log(rng, 1100, 100000)
    elif kind == "synth":
        c["npix"] = _log(rng, 100, 60000)
        c["nl"] = rng.choice([rng.randint(6, 32), rng.randint(33, 100)])
        c["precision"] = rng.choice(["fp32", "fp32", "fp64"])
    elif kind == "fits":
        c["npix"] = 16 * _log(rng, 100, 4000)
        c["nl"] = rng.randint(5, 60)
        c["order"] = rng.choice(["LSRC", "LRSC", "RCLS", "RCSL"])
    elif kind == "mac":
        c["npix"] = _log(rng, 200, 12000)
        c["slight"], c["mac"] = "shared", True
    elif kind == "fp64":
        c["npix"] = _log(rng, 100, 6000)
        c["precision"] = "fp64"
    elif kind == "lm_mils":
        c["npix"] = 1
    elif kind == "server":
        c["npix"], c["scans"], c["nl"] = _log(rng, 500, 20000), rng.randint(2, 9), 30
        c["fwhm"] = 60.0
    return c


# ---- the physics in 64 bits, for inputs and for exact() ----
VLIGHT, ZEEMAN, RSQRTPI = 2.99792458e5, 4.6686411e-13, 0.5641895836
P6 = (122.607931777104326, 214.382388694706425, 181.928533092181549, 93.155580458138441, 30.180142196210589,
      5.912626209773153, 0.564189583562615)
Q7 = (122.60793177387535, 352.730625110963558, 457.334478783897737, 348.703917719495792, 170.354001821091472,
      53.992906912940207, 10.479857114260399)


def grid(nl, lambda0):
    """Offsets [mA] and wavelengths [A] around the line, its centre on the middle sample."""
    step = 21.5 if nl > 32 else round(725.0 / (nl - 1), 1) if nl > 8 else 69.0
    offs = (np.arange(nl) - nl // 2) * step
    return offs, lambda0 + offs / 1000.0


def voigt(a, u):
    """H and F (half the imaginary part) of the Voigt and Faraday-Voigt functions."""
    z = torch.complex(a.expand_as(u), -u)
    num = torch.full_like(z, P6[6])
    for c in P6[5::-1]:
        num = num * z + c
    den = z + Q7[6]
    for c in Q7[5::-1]:
        den = den * z + c
    w = num / den
    return w.real, w.imag / 2


def zeeman(line):
    """Splittings and strengths of the pi, blue and red groups."""
    c = line._c
    blue = [c.nub[k] for k in range(c.n_sig)]
    return [([c.nup[k] for k in range(c.n_pi)], [c.wep[k] for k in range(c.n_pi)]),
            (blue, [c.web[k] for k in range(c.n_sig)]),
            ([-x for x in blue[::-1]], [c.wer[k] for k in range(c.n_sig)])]


def correlation(psf, nl, dev):
    """out = x @ M.T of the instrumental profile over a grid, zeros beyond it."""
    M = np.zeros((nl, nl))
    for k in range(nl):
        for i in range(nl):
            if 0 <= i - k + nl // 2 < nl:
                M[k, i] = psf[i - k + nl // 2]
    return torch.as_tensor(M, device=dev)


def instrument(x, M):
    """x [n][4][...][nl]: of Stokes I the depth below the continuum is correlated."""
    i = x[:, :1]
    ic = torch.maximum(i[..., :1], i[..., -1:])
    return torch.cat([ic - (ic - i) @ M.T, x[:, 1:] @ M.T], dim=1)


def profiles(line, lam, m, rf=False):
    """Stokes profiles [n][4][nl] of models [n][11] before the instrument, and
    with rf their response functions [n][4][9][nl]."""
    lam = torch.as_tensor(lam, device=m.device)
    p = [m[:, i:i + 1] for i in range(11)]
    rad = math.pi / 180.0
    l0, E0, LD, A = line.lambda0, p[0] * line._c.fo, p[3], p[4]
    si, ci = torch.sin(p[5] * rad), torch.cos(p[5] * rad)
    s2, c2 = torch.sin(2 * p[6] * rad), torch.cos(2 * p[6] * rad)
    u = (lam - l0) / LD - p[2] * l0 / (VLIGHT * LD)
    per_gauss = l0 * l0 * ZEEMAN / LD
    fi, shi, dfi, dshi = [], [], [], []
    for nu, we in zeeman(line):
        f, h, last = 0.0, 0.0, None
        for n, w in zip(nu, we):
            uu = u - per_gauss * n * p[1]
            H, F = voigt(A, uu)
            f, h = f + w * H, h + 2 * w * F
            last = (n, w, uu, H, F)
        fi.append(f)
        shi.append(h)
        if rf:  # the last component's derivatives in B, v_los, Doppler width and damping
            n, w, uu, H, F = last
            dHu, dFu = (4 * A * F - 2 * uu * H) * w, (RSQRTPI - A * H - 2 * uu * F) * w
            chain = (-per_gauss * n, -l0 / (VLIGHT * LD), -uu / LD)
            dfi.append([dHu * c for c in chain] + [-2 * dFu])
            dshi.append([dFu * c for c in chain] + [dHu / 2])

    def matrix(f, h, e, si2, cross, cosi, cc, ss):
        """eta_I, Q, U, V and rho_Q, U, V of strength e."""
        d, r = f[0] - (f[1] + f[2]) / 2, h[0] - (h[1] + h[2]) / 2
        return (e / 2 * (f[0] * si2 + (f[1] + f[2]) * cross), e / 2 * d * cc, e / 2 * d * ss,
                e / 2 * (f[2] - f[1]) * cosi, e / 2 * r * cc, e / 2 * r * ss, e / 2 * (h[2] - h[1]) * cosi)

    angles = (si * si, (1 + ci * ci) / 2, ci, si * si * c2, si * si * s2)
    eta = matrix(fi, shi, E0, *angles)
    e, q, uq, v, rq, ru, rv = (1 + eta[0],) + eta[1:]
    gp1 = e * e - q * q - uq * uq - v * v + rq * rq + ru * ru + rv * rv
    gp2 = q * rq + uq * ru + v * rv
    gp3 = e * e + rq * rq + ru * ru + rv * rv
    det = e * e * gp1 - gp2 * gp2
    g = (e * e * q + e * (v * ru - uq * rv) + rq * gp2, e * e * uq + e * (q * rv - v * rq) + ru * gp2,
         e * e * v + e * (uq * rq - q * ru) + rv * gp2)
    b1 = -p[8]
    S = torch.stack([p[7] - b1 / det * e * gp3] + [b1 / det * x for x in g], dim=1)
    if not rf:
        return S, None
    one = [matrix(fi, shi, torch.ones_like(E0), *angles)]
    for k in range(4):
        one.append(matrix([d[k] for d in dfi], [d[k] for d in dshi], E0, *angles))
    one.append(matrix(fi, shi, E0, 2 * rad * si * ci, -rad * si * ci, -rad * si, 2 * rad * si * ci * c2,
                      2 * rad * si * ci * s2))
    one.append(matrix(fi, shi, E0, 0 * si, 0 * si, 0 * si, -2 * rad * si * si * s2, 2 * rad * si * si * c2))
    rows = []
    for de, dq, du, dv, drq, dru, drv in one:
        d1 = 2 * (e * de - q * dq - uq * du - v * dv + rq * drq + ru * dru + rv * drv)
        d2 = rq * dq + q * drq + ru * du + uq * dru + rv * dv + v * drv
        d3 = 2 * (e * de + rq * drq + ru * dru + rv * drv)
        dd = 2 * e * de * gp1 + e * e * d1 - 2 * gp2 * d2
        dg = (2 * e * de * q + e * e * dq + de * (v * ru - uq * rv) + e * (dv * ru + v * dru - du * rv - uq * drv)
              + drq * gp2 + rq * d2,
              2 * e * de * uq + e * e * du + de * (q * rv - v * rq) + e * (dq * rv + q * drv - dv * rq - v * drq)
              + dru * gp2 + ru * d2,
              2 * e * de * v + e * e * dv + de * (uq * rq - q * ru) + e * (du * rq + uq * drq - dq * ru - q * dru)
              + drv * gp2 + rv * d2)
        k = b1 / (det * det)
        rows.append(torch.stack([-k * ((de * gp3 + e * d3) * det - dd * e * gp3)]
                                + [k * (x * det - dd * y) for x, y in zip(dg, g)], dim=1))
    rows.append(torch.zeros_like(S))
    rows[7][:, 0] = 1.0
    rows.append(torch.stack([e * gp3 / det] + [-x / det for x in g], dim=1))
    return S, torch.stack(rows, dim=2)


def _line(case):
    l0, quantum = LINES[case["line"]]
    return pm.LineData(specs.FE6302 if case["nl"] > 32 and case["line"] == "triplet" else l0, quantum)


def _setup(case, nl=None):
    """Line, wavelengths, taps, NTERMS, fix[] and the initial guess of a case."""
    line = _line(case)
    offs, lam = grid(nl or case["nl"], line.lambda0)
    psf = pm.psf_gaussian(case["fwhm"], lam) if case["fwhm"] else None
    nterms, fix, guess = specs.nterms_fix_guess(2 if case["slight"] != "none" else 1)
    if case["mac"]:
        nterms, fix = 11, [1] * 11
        guess[9] = 1.0
    return line, lam, psf, nterms, fix, guess


def _models(case, seed, n):
    rng = np.random.default_rng(seed)
    m = specs.truth_models(2 if case["slight"] != "none" else 1, n, rng)
    if case["mac"]:
        m[:, 9] = rng.uniform(0.3, 2.0, n)
    return m


def _quiet(line, lam, psf):
    """The stray-light profile [4][nl]: a quiet-Sun atmosphere through the instrument."""
    m = torch.as_tensor(specs.QUIET_SUN_B0[None, :], device="cuda")
    S, _ = profiles(line, lam, m)
    if psf is not None:
        S = instrument(S, correlation(psf, len(lam), "cuda"))
    return S[0].float()


def _observed(case, seed, n, line, lam, psf, sl=None):
    """Observed profiles [n][4][nl] float32 on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    m = torch.as_tensor(_models(case, seed, n), device="cuda")
    M = None if psf is None else correlation(psf, len(lam), "cuda")
    x = torch.as_tensor(lam - lam[len(lam) // 2], device="cuda")
    obs = torch.empty((n, 4, len(lam)), dtype=torch.float32, device="cuda")
    for a in range(0, n, 32768):
        p = m[a:a + 32768]
        S, _ = profiles(line, lam, p)
        if case["mac"]:
            k = torch.exp(-0.5 * ((x[None, :] - x[:, None])[None] * VLIGHT / (line.lambda0 * p[:, 9, None, None])) ** 2)
            S = torch.einsum("nsi,nki->nsk", S, k / k.sum(dim=2, keepdim=True))
        if M is not None:
            S = instrument(S, M)
        if sl is not None:
            S = S * p[:, 10, None, None] + sl.double() * (1 - p[:, 10, None, None])
        noise = torch.randn(S.shape, generator=g, device="cuda", dtype=torch.float64)
        obs[a:a + 32768] = (S + specs.NOISE_SIGMA * noise).float()
    return obs


def _pinned(n, nl):
    pin = lambda shape, dt: torch.empty(shape, dtype=dt, pin_memory=True).numpy()  # noqa: E731
    return {"models": pin((n, 11), torch.float64), "chisq": pin((n,), torch.float32),
            "iters": pin((n,), torch.int32)}


def _fits(case, seed):
    """The bytes of a FITS spectro cube: header and big-endian float32 data."""
    nl, rows = case["nl"], case["npix"] // 250 if case["npix"] % 250 == 0 else 16
    size = {"L": nl, "S": 4, "R": rows, "C": case["npix"] // rows}
    role = {"L": "WAVE-GRI", "S": "STOKES", "R": "HPLN-TAN", "C": "HPLT-TAN"}
    order = case["order"]
    cards = ["SIMPLE  =                    T", "BITPIX  =                  -32", "NAXIS   =                    4"]
    cards += ["NAXIS%d  = %20d" % (i + 1, size[r]) for i, r in enumerate(order)]
    cards += ["CTYPE%d  = '%-8s'" % (i + 1, role[r]) for i, r in enumerate(order)] + ["END"]
    head = "".join("%-80s" % c for c in cards).encode()
    head += b" " * (-len(head) % 2880)
    data = np.random.default_rng(seed).standard_normal([size[r] for r in order[::-1]], dtype=np.float32)
    body = data.astype(">f4").tobytes()
    return head + body + b"\0" * (-len(body) % 2880), data


def prepare(case, seed):
    kind, n = case["kind"], case["npix"]
    s = {"case": case}
    if kind == "fits":
        s["bytes"], _ = _fits(case, seed)
        return s
    prec = pm.PREC_FP32 if case["precision"] == "fp32" else pm.PREC_FP64
    line, lam, psf, nterms, fix, guess = _setup(case)
    s["guess"] = guess
    if kind == "server":
        grids, s["scans"] = [], []
        for i, nl in enumerate(SERVER_GRIDS):
            gl, glam, gpsf, _, _, _ = _setup(case, nl)
            grids.append(pm.Grid(lam=glam, psf=gpsf, guess=guess, noise=NOISE))
        for k in range(case["scans"]):
            i = k % len(SERVER_GRIDS)
            obs = _observed(case, 64 * int(seed) + k, n, line, grids[i].lam, grids[i].psf)
            host = torch.empty(obs.shape, dtype=torch.float32, pin_memory=True)
            s["scans"].append((i, host.copy_(obs).numpy()))
        s["server"] = pm.Server(line, grids, hbm_budget_bytes=1 << 30, linger_ms=0.5)
        return s
    s["inv"] = pm.Inverter(line, lam, psf, noise=NOISE, fix=fix, nterms=nterms, precision=prec)
    if kind == "synth":
        s["models"] = torch.as_tensor(_models(case, seed, n), device="cuda")
        return s
    sl = None if case["slight"] == "none" else _quiet(line, lam, psf)
    s["obs"] = _observed(case, seed, n, line, lam, psf, sl)
    s["slight"] = sl
    if case["slight"] == "pixel":
        s["slight"] = sl[None].expand(n, 4, case["nl"]).contiguous()
    if kind != "device":
        s["slight"] = None if sl is None else s["slight"].cpu().numpy()
        host = torch.empty(s["obs"].shape, dtype=torch.float32, pin_memory=kind == "pinned")
        s["obs"] = host.copy_(s["obs"]).numpy()
        if kind == "pinned":
            s["out"] = _pinned(n, case["nl"])
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "lm_mils":
        rc, model, spectra, chisq, iters = s["inv"].lm_mils(s["obs"][0], s["guess"])
        return {"rc": rc, "model": model, "spectra": spectra, "chisq": np.float32(chisq), "iters": iters}
    if kind == "device":
        return s["inv"].invert(s["obs"], s["guess"], slight=s["slight"])
    if kind == "host":
        return s["inv"].invert(s["obs"], s["guess"], slight=s["slight"])
    if kind == "pinned":
        return s["inv"].invert(s["obs"], s["guess"], want_spectra=False, want_status=False, out=s["out"])
    if kind == "synth":
        spectra, rf = s["inv"].synth(s["models"], rf=True)
        return {"spectra": spectra, "rf": rf}
    if kind == "server":
        ids = [s["server"].submit(g, obs) for g, obs in s["scans"]]
        done = [s["server"].wait(i) for i in ids]
        return [{k: d[k] for k in ("models", "chisq", "iters", "status")} for d in done]
    return pm.ingest_fits(s["bytes"])


def _flops(nl, K, steps, accepted, taps):
    """The frozen count of one pixel: synthesis, response functions with normal
    equations, chi^2 and the FP64 solve (add, sub, mul, div 1; FMA 2)."""
    syn = nl * 400 + 8 * nl * taps
    resp = 870 * nl + 8 * nl * taps * (K - 1)
    normal = 4 * nl * (K * K + 3 * K)
    solve = 9 * K ** 3 + 4 * K * K
    if not steps:
        return syn + resp
    return (1 + steps) * (syn + 20 * nl) + (1 + accepted) * (resp + normal) + steps * solve


def work(case):
    n, nl = case["npix"], case["nl"]
    if case["kind"] == "fits":
        return {"bytes": 2.0 * 16 * n * nl, "flops": 0.0}
    K = 11 if case["mac"] else 10 if case["slight"] != "none" else 9
    if case["kind"] == "synth":
        return {"bytes": n * (88.0 + 16 * nl * (1 + K)), "flops": float(n) * _flops(nl, K, 0, 0, min(nl, 32))}
    out = 88 + 8 + (4 + 16 * nl if case["kind"] not in ("pinned", "server") else 0)
    if case["kind"] == "server":
        sizes = [SERVER_GRIDS[k % 3] for k in range(case["scans"])]
        return {"bytes": float(sum(n * (16 * m + out) for m in sizes)),
                "flops": float(sum(n * _flops(m, K, STEPS, ACCEPTED, m) for m in sizes))}
    taps = 0 if not case["fwhm"] else nl if nl <= 32 else 9
    return {"bytes": n * (16.0 * nl * (2 if case["slight"] == "pixel" else 1) + out),
            "flops": float(n) * _flops(nl, K, STEPS, ACCEPTED, taps)}


def exact(case, seed):
    """The synthesized profiles and response functions, or the file's values, in
    64 bits.  An inversion has none: it ends where its own arithmetic's rounding
    lets the iteration end, on the noise floor of its profiles."""
    if case["kind"] == "fits":
        _, data = _fits(case, seed)
        at = case["order"][::-1].index
        cube = data.transpose(at("C"), at("R"), at("S"), at("L"))
        return torch.as_tensor(cube.reshape(case["npix"], 4, case["nl"]).astype(np.float64))
    if case["kind"] != "synth":
        return None
    line, lam, psf, nterms, _, _ = _setup(case)
    m = torch.as_tensor(_models(case, seed, case["npix"]), device="cuda")
    M = None if psf is None else correlation(psf, case["nl"], "cuda")
    spectra, rf = [], []
    for a in range(0, case["npix"], 8192):
        S, R = profiles(line, lam, m[a:a + 8192], rf=True)
        if M is not None:
            R = torch.cat([instrument(R[:, :, :7], M), R[:, :, 7:8], instrument(R[:, :, 8:], M)], dim=2)
            S = instrument(S, M)
        spectra.append(S)
        rf.append(R)
    return {"spectra": torch.cat(spectra), "rf": torch.cat(rf)}
