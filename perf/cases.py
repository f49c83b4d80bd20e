"""Timed cases of the passive forward path and of the T-matrix branch.

Each case is one call of a public entry point as a user's program makes it:
``pyPamtra.runPamtra`` (a profile on the host, passive and simple radar),
``batch.run`` (packed columns resident on the device), ``batch.run_host``
(packed columns in page-locked host memory) and ``tmatrix.calc_tmatrix_batch``
(size bins of spheroids on the device).  Workloads are seeded synthetic
columns of the shapes in ``pamtra_b200/workloads.py``.

``exact`` holds a plain numpy restatement of the path for liquid clouds and
rain, used for the cases with few columns.
"""

import math
import warnings

import numpy as np
import torch

from pamtra_b200 import batch, core, meteoSI, tmatrix, workloads
from pamtra_b200._native import PREC_3XTF32, PREC_FP64, PREC_FP64_BATCHED

PRECISIONS = {"fp64": PREC_FP64, "fp64_batched": PREC_FP64_BATCHED, "3xtf32": PREC_3XTF32}
# window and sounding channels of microwave radiometers (GHz), ascending
CHANNELS = [10.65, 18.7, 23.8, 31.4, 36.5, 89.0, 150.0, 183.31]
EXACT_COLUMNS = 2  # columns up to which the numpy restatement takes seconds


def listed():
    return [
        # one profile through the session object, the way most scripts start
        dict(name="profile", entry="profile", cols=1, layers=50, freqs=2),
        # one column already on the device: launch latency and serial chains
        dict(name="column", entry="device", kind="cloud_rain", precision="fp64", cols=1, layers=50, freqs=3, nummu=16),
        # a handful of columns (a radiometer's time series of one hour)
        dict(name="columns_24", entry="device", kind="cloud_rain", precision="fp64_batched", cols=24, layers=50, freqs=4,
             nummu=16),
        # a model slice: the throughput shape
        dict(name="columns_1500", entry="device", kind="cloud_rain", precision="fp64_batched", cols=1500, layers=50,
             freqs=4, nummu=16),
        # the same shape in the split-precision form
        dict(name="split_1024", entry="device", kind="cloud_rain", precision="3xtf32", cols=1024, layers=50, freqs=4,
             nummu=16),
        # end to end from page-locked host buffers
        dict(name="host_333", entry="host", kind="cloud_rain", precision="fp64_batched", cols=333, layers=50, freqs=4,
             nummu=16),
        # tall columns with ice, snow, cloud water and rain
        dict(name="tall_64", entry="device", kind="tall", precision="fp64_batched", cols=64),
        # mixed requests: own layers, species, frequencies and NUMMU 8/16/32 per column
        dict(name="uneven_40", entry="device", kind="uneven", precision="fp64_batched", cols=40, freqs=20),
        dict(name="uneven_split_40", entry="device", kind="uneven", precision="3xtf32", cols=40, freqs=20),
        # long size spectra at high frequencies: single scattering dominates
        dict(name="mie_heavy_40", entry="device", kind="mie_heavy", precision="fp64_batched", cols=40),
        # T-matrix of upright and of canted spheroids
        dict(name="tmatrix_32x32", entry="tmatrix", items=32, bins=32, canted=False, nummu=16),
        dict(name="tmatrix_canted_3x32", entry="tmatrix", items=3, bins=32, canted=True, nummu=16),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    which = rng.choice(["profile", "device", "device", "device", "host", "tall", "uneven", "mie_heavy", "tmatrix", "canted"])
    prec = rng.choice(["fp64", "fp64_batched", "fp64_batched", "3xtf32"])
    if which == "profile":
        return dict(entry="profile", cols=_log_int(rng, 1, 40), layers=rng.randint(20, 120), freqs=rng.randint(1, 8))
    if which in ("device", "host"):
        nummu = rng.choice([8, 16, 16, 32])
        layers, freqs = rng.randint(20, 120), rng.randint(1, 8)
        most = max(1, int(1400 * 200 / (layers * freqs) / (8 if nummu == 32 else 1)))
        return dict(entry=which, kind="cloud_rain", precision=prec, cols=_log_int(rng, 1, most), layers=layers,
                    freqs=freqs, nummu=nummu)
    if which == "uneven":
        return dict(entry="device", kind="uneven", precision=prec, cols=_log_int(rng, 3, 40), freqs=rng.randint(4, 20))
    if which in ("tall", "mie_heavy"):
        return dict(entry="device", kind=which, precision=prec, cols=_log_int(rng, 1, 64 if which == "tall" else 40))
    if which == "tmatrix":
        return dict(entry="tmatrix", items=_log_int(rng, 1, 60), bins=rng.randint(11, 50), canted=False,
                    nummu=rng.choice([8, 16, 16, 32]))
    return dict(entry="tmatrix", items=rng.randint(1, 4), bins=rng.randint(7, 32), canted=True, nummu=rng.choice([8, 16]))


# ------------------------------------------------------------------ inputs
def _cloud_rain(case, seed):
    """Columns over 0-12 km of a jittered standard atmosphere with cloud
    liquid and rain between 1.2 and 6.2 km, mixing ratios log-uniform over
    0.01-2 g/kg."""
    warnings.simplefilter("ignore")
    rng = np.random.default_rng(seed)
    n, nl = case["cols"], case["layers"]
    z = np.linspace(0.0, 12000.0, nl + 1)
    _, p0, t0 = meteoSI.usStandard(z)
    pam = core.pyPamtra()
    pam.df.addHydrometeor(workloads.CLOUD_C1)
    pam.df.addHydrometeor(workloads.RAIN_C1)
    pam.nmlSet["hydro_adaptive_grid"] = False
    pam.nmlSet["emissivity"] = 0.5
    band = (0.5 * (z[1:] + z[:-1]) > 1200.0) & (0.5 * (z[1:] + z[:-1]) < 6240.0)
    q = 10.0 ** rng.uniform(-5.0, math.log10(2e-3), (n, 1, nl, 2)) * band[None, None, :, None]
    pam.createProfile(hgt_lev=np.tile(z, (n, 1, 1)),
                      temp_lev=t0 + rng.uniform(-1.0, 1.0, (n, 1, nl + 1)),
                      press_lev=p0 * (1.0 + rng.uniform(-0.005, 0.005, (n, 1, nl + 1))),
                      relhum_lev=rng.uniform(40.0, 95.0, (n, 1, nl + 1)),
                      hydro_q=q, groundtemp=290.0, sfc_refl="S", obs_height=np.tile([833000.0, 0.0], (n, 1, 1)))
    return pam


def _channels(n):
    """``n`` ascending frequencies spread over the channels."""
    return sorted(CHANNELS[(3 * i + 2) % len(CHANNELS)] for i in range(n))


def _pack(case, seed):
    if case["kind"] == "cloud_rain":
        return batch.pack_pam(_cloud_rain(case, seed), _channels(case["freqs"]), nummu=case["nummu"])
    if case["kind"] == "uneven":
        n, f = case["cols"], case["freqs"]  # the three NUMMU as three requests merged into one batch
        parts = [(n - 2 * (n // 3), 8, f), (n // 3, 16, (f + 1) // 2), (n // 3, 32, (3 * f + 3) // 4)]
        return batch.concat([workloads.uneven_batch(c, seed=3 * seed + i, nummu_choices=(nummu,), nfreq_range=(k, k))
                             for i, (c, nummu, k) in enumerate(parts)])[0]
    if case["kind"] == "tall":
        return workloads.target_batch(case["cols"], seed=seed)
    return workloads.mie_heavy_batch(case["cols"], seed=seed)


def _spheroids(case, seed):
    """Soft ice spheroids (snow and graupel aggregates) of 0.2-4 mm with
    exponential spectra, one frequency per item."""
    rng = np.random.default_rng(seed)
    ni, nb = case["items"], case["bins"]
    edges = np.linspace(0.2e-3, 4e-3, nb + 1) * rng.uniform(0.9, 1.1, (ni, 1))
    d = 0.5 * (edges[:, 1:] + edges[:, :-1])
    n = 10.0 ** rng.uniform(6.0, 8.0, (ni, 1)) * np.exp(-d * rng.uniform(1e3, 3e3, (ni, 1)))
    a = dict(dmax=d, del_d=np.diff(edges, axis=1), ndens=n, density=np.tile(rng.uniform(100.0, 600.0, (ni, 1)), nb),
             as_ratio=np.tile(rng.uniform(0.5, 0.9, (ni, 1)), nb),
             canting=np.tile(rng.uniform(5.0, 40.0, (ni, 1)), nb) if case["canted"] else np.zeros((ni, nb)))
    args = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in a.items()}
    args["freq"] = torch.from_numpy(rng.choice([35.5e9, 89.0e9, 157.0e9], ni)).cuda()
    args["ref_index"] = torch.from_numpy(1.78 - 1j * rng.uniform(1e-3, 4e-3, ni)).cuda()
    args["phase"] = torch.full((ni,), -1, dtype=torch.int32, device="cuda")
    return args


def prepare(case, seed):
    entry = case["entry"]
    if entry == "tmatrix":
        return dict(entry=entry, args=_spheroids(case, seed), nummu=case["nummu"])
    if entry == "profile":
        return dict(entry=entry, pam=_cloud_rain(case, seed), freqs=_channels(case["freqs"]))
    b = _pack(case, seed)
    if entry == "host":
        b.pinned_arrays()
        out = b.alloc_outputs(None, pinned=True)
    else:
        b.device_arrays(torch.device("cuda", 0))
        out = b.alloc_outputs(torch.device("cuda", 0))
    return dict(entry=entry, batch=b, out=out, precision=PRECISIONS[case["precision"]])


def run(state):
    entry = state["entry"]
    if entry == "profile":
        pam = state["pam"]
        pam.runPamtra(state["freqs"])
        return {k: pam.r[k] for k in ("tb", "emissivity", "angles_deg", "status", "Ze", "Att_hydro", "Att_atmo")}
    if entry == "tmatrix":
        o = tmatrix.calc_tmatrix_batch(nummu=state["nummu"], **state["args"])
        return {k: o[k] for k in tmatrix.OUT_KEYS}
    call = batch.run_host if entry == "host" else batch.run
    return call(state["batch"], outputs=state["out"], precision=state["precision"])


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: inputs and outputs once.  Operations: per scattering (layer,
    frequency) 14 doublings and one adding step, with the products of n x n
    matrices (n = 2 NUMMU) that symmetric R and T leave (four and six), and
    the Mie sums over bins, terms and angles; for a T-matrix bin one solve
    per azimuthal order and the angular sums."""
    if case["entry"] == "tmatrix":
        nb, n = case["items"] * case["bins"], case["nummu"]
        solve = 10 * 8 * (2 * 10) ** 3 / 3
        angular = n * 2 * n * 30 * 10 * 16 * (10 if case["canted"] else 1)
        return dict(bytes=nb * 56.0 + case["items"] * (8 * n * n + 6 * n + 4) * 8.0 + nb * 12.0, flops=nb * (solve + angular))
    cols = case["cols"]
    kind = case.get("kind", "cloud_rain")
    layers, scat, freqs, nsp, bins, terms, n = {
        "cloud_rain": (case.get("layers", 50), 0.42 * case.get("layers", 50), case.get("freqs", 4), 2, 45, 12,
                       2 * case.get("nummu", 16)),
        "uneven": (95, 60, 0.75 * case.get("freqs", 20), 5, 50, 12, 38), "tall": (150, 140, 4, 4, 40, 12, 32),
        "mie_heavy": (100, 90, 4, 4, 200, 15, 32)}[kind]
    doubling, adding = 14 * 4 * 2.0 * n ** 3, 6 * 2.0 * n ** 3
    mie = 0.6 * nsp * bins * terms * (3 * terms) * 8.0
    nbytes = cols * (layers * (8 + 3 * nsp) * 8.0 + freqs * (2 * n * 2 * 8.0 + n * 8.0 + 4))
    return dict(bytes=nbytes, flops=cols * freqs * scat * (doubling + adding + mie))


# ------------------------------------------------------------------ numpy restatement
_O2_F = np.array("""118.7503 56.2648 62.4863 58.4466 60.3061 59.5910 59.1642 60.4348 58.3239 61.1506 57.6125 61.8002
56.9682 62.4112 56.3634 62.9980 55.7838 63.5685 55.2214 64.1278 54.6712 64.6789 54.1300 65.2241 53.5957 65.7648 53.0669
66.3021 52.5424 66.8368 52.0214 67.3696 51.5034 67.9009 368.4984 424.7631 487.2494 715.3932 773.8397 834.1453""".split(),
                 dtype=np.float64)
_O2_S = 1e-15 * np.array("""2.936 .8079 2.480 2.228 3.351 3.292 3.721 3.891 3.640 4.005 3.227 3.715 2.627 3.156 1.982
2.477 1.391 1.808 .9124 1.230 .5603 .7842 .3228 .4689 .1748 .2632 .08898 .1389 .04264 .06899 .01924 .03229 .008191 .01423
.6460 7.047 3.011 1.826 11.52 3.971""".split(), dtype=np.float64)
_O2_B = np.array(""".009 .015 .083 .084 .212 .212 .391 .391 .626 .626 .915 .915 1.26 1.26 1.66 1.665 2.119 2.115 2.624
2.625 3.194 3.194 3.814 3.814 4.484 4.484 5.224 5.224 6.004 6.004 6.844 6.844 7.744 7.744 .048 .044 .049 .145 .141
.145""".split(), dtype=np.float64)
_O2_W = np.array("""1.63 1.646 1.468 1.449 1.382 1.360 1.319 1.297 1.266 1.248 1.221 1.207 1.181 1.171 1.144 1.139 1.110
1.108 1.079 1.078 1.05 1.05 1.02 1.02 1.0 1.0 .97 .97 .94 .94 .92 .92 .89 .89 1.92 1.92 1.92 1.81 1.81 1.81""".split(),
                 dtype=np.float64)
_O2_Y = np.array("""-.0233 .2408 -.3486 .5227 -.5430 .5877 -.3970 .3237 -.1348 .0311 .0725 -.1663 .2832 -.3629 .3970
-.4599 .4695 -.5199 .5187 -.5597 .5903 -.6246 .6656 -.6942 .7086 -.7325 .7348 -.7546 .7702 -.7864 .8083 -.8210 .8439
-.8529 0 0 0 0 0 0""".split(), dtype=np.float64)
_O2_V = np.array(""".0079 -.0978 .0844 -.1273 .0699 -.0776 .2309 -.2825 .0436 -.0584 .6056 -.6619 .6451 -.6759 .6547
-.6675 .6135 -.6139 .2952 -.2895 .2654 -.2590 .3750 -.3680 .5085 -.5002 .6206 -.6091 .6526 -.6393 .6640 -.6475 .6729
-.6545 0 0 0 0 0 0""".split(), dtype=np.float64)
# line centre, strength, temperature exponent, dry width and its exponent, self width and its exponent
_H2O = np.array("""22.2351 .1310e-13 2.144 .002656 .69 .0127488 .61
183.3101 .2273e-11 .668 .00281 .64 .01491 .85
321.2256 .8036e-13 6.179 .0023 .67 .0108 .54
325.1529 .2694e-11 1.541 .00278 .68 .0135 .74
380.1974 .2438e-10 1.048 .00287 .54 .01541 .89
439.1508 .2179e-11 3.595 .0021 .63 .0090 .52
443.0183 .4624e-12 5.048 .00186 .60 .00788 .50
448.0011 .2562e-10 1.405 .00263 .66 .01275 .67
470.8890 .8369e-12 3.597 .00215 .66 .00983 .65
474.6891 .3263e-11 2.379 .00236 .65 .01095 .64
488.4911 .6659e-12 2.852 .0026 .69 .01313 .72
556.9360 .1531e-08 .159 .00321 .69 .01320 1.0
620.7008 .1707e-10 2.391 .00244 .71 .01140 .68
752.0332 .1011e-08 .396 .00306 .68 .01253 .84
916.1712 .4227e-10 1.441 .00267 .70 .01275 .78""".split(), dtype=np.float64).reshape(15, 7).T
_C, _RD, _RV = 299792458.0, 287.0596736665907, 461.5249933083879


def _gas(f, t, rho_vap, press):
    """Rosenkranz-98 absorption (1/m) of layers."""
    p, rho, th = press / 100.0, rho_vap * 1e3, 300.0 / t
    pwv = rho * t / 217.0
    pda = p - pwv
    den = 0.001 * (pda * th ** 0.8 + 1.1 * pwv * th)
    w = 0.56 * den
    s = 1.6e-17 * f * f * w / (th * (f * f + w * w))
    for fk, sk, bk, wk, yk, vk in zip(_O2_F, _O2_S, _O2_B, _O2_W, _O2_Y, _O2_V):
        df = wk * den
        y = 0.001 * p * th ** 0.8 * (yk + vk * (th - 1))
        s = s + sk * np.exp(-bk * (th - 1)) * (f / fk) ** 2 * ((df + (f - fk) * y) / ((f - fk) ** 2 + df * df) +
                                                            (df - (f + fk) * y) / ((f + fk) ** 2 + df * df))
    air = 0.5034e12 * s * pda * th ** 3 / np.pi + 6.4e-14 * p * p * f * f * th ** 3.55
    s = 0.0
    for fl, s1, b2, w3, x, ws, xs in _H2O.T:
        w = w3 * pda * th ** x + ws * pwv * th ** xs
        res = sum(w / (d * d + w * w) - w / (562500.0 + w * w) for d in (f - fl, f + fl) if abs(d) < 750.0)
        s = s + s1 * th ** 2.5 * np.exp(b2 * (1 - th)) * res * (f / fl) ** 2
    con = (5.43e-10 * 1.105 * pda * th ** 3 + 1.8e-8 * 0.79 * pwv * th ** 7.5) * pwv * f * f
    return (air + 0.3183e-4 * 3.335e16 * rho * s + con) / 1e3


def _water(t, f):
    """Refractive index of water (Turner, Kneifel and Cadeddu)."""
    tc, w = t - 273.15, 2e9 * np.pi * f
    es = 87.9144 - 0.404399 * tc + 9.58726e-4 * tc ** 2 - 1.32802e-6 * tc ** 3
    re, im = es, 0.0
    for a, b, c, d in ((81.69396, 4.410555e-3, 1.208992e-13, 676.8769), (1.597733, 1.060228e-2, 9.982113e-15, 572.0517)):
        tau, dl = c * np.exp(d / (tc + 135.1758)), a * np.exp(-b * tc)
        re = re - (w * tau) ** 2 * dl / (1 + (w * tau) ** 2)
        im = im + w * tau * dl / (1 + (w * tau) ** 2)
    return np.sqrt(re + 1j * im)


def _bins(row, q):
    """Bin centres, widths and particles per volume of an exponential spectrum
    holding ``q`` kg/m3 in each layer."""
    nbin, p2, n0, lo, hi = int(row[9]), row[12], row[13], row[15] + 1e-8, row[16]
    half = nbin // 2
    lin = half - 1 if 2 * half == nbin else half
    e = np.sort(np.concatenate([lo + (hi - lo) / (lin + 1) * np.arange(1, lin + 2),
                                lo * (hi / lo) ** (np.arange(half + 1) / (half + 1.0))]))
    am = 1000.0 * np.pi / 6
    if p2 > 0:
        lam = np.full_like(q, 3.0 / p2)
        n0 = q * lam ** 4 / (am * 6.0)
    else:
        lam = (n0 * am * 6.0 / q) ** 0.25
        n0 = np.full_like(q, n0)
    g = n0[:, None] * np.exp(-lam[:, None] * e)
    d, dd = 0.5 * (e[1:] + e[:-1]), np.diff(e)
    n = 0.5 * (g[:, 1:] + g[:, :-1]) * dd
    n = n * (q / np.sum(am * n * d ** 3, axis=1))[:, None]
    n[n < n.sum(1, keepdims=True) / nbin * 1e-60] = 0.0
    return d, dd, n


def _mie(f, d, n, m):
    """Extinction, scattering and backscattering of layers and the Legendre
    coefficients [layer][3][l] of P11, P12, P33."""
    wl = _C / (f * 1e9)
    x = np.pi * d / wl
    stop = (x + 4.0 * x ** float(np.float32(0.3334)) + 2).astype(int)
    top, k = int(stop[-1]), int(stop.max())
    y = m[:, None] * x
    mm = m[:, None]
    D = np.zeros((k + 17,) + y.shape, dtype=complex)
    for j in range(k + 16, 1, -1):
        D[j - 1] = j / y - 1.0 / (D[j] + j / y)
    pm, p, cm, c = np.cos(x), np.sin(x), -np.sin(x), np.cos(x)
    a, b = np.zeros((2, k + 1) + y.shape, dtype=complex)
    for j in range(1, k + 1):
        pm, p = p, (2 * j - 1) / x * p - pm
        cm, c = c, (2 * j - 1) / x * c - cm
        on = stop >= j
        for o, t in ((a, D[j] / mm + j / x), (b, D[j] * mm + j / x)):
            o[j] = np.where(on, (t * p - pm) / (t * (p - 1j * c) - (pm - 1j * cm)), 0.0)
    j = np.arange(k + 1)[:, None, None]
    area = np.pi * (d / 2) ** 2
    qe = 2 / x ** 2 * np.sum((2 * j + 1) * (a + b).real, 0)
    qs = 2 / x ** 2 * np.sum((2 * j + 1) * (abs(a) ** 2 + abs(b) ** 2), 0)
    qb = abs(np.sum((2 * j + 1) * (-1.0) ** j * (a - b), 0)) ** 2 / x ** 2
    ext, sca, back = ((v * area * n).sum(1) for v in (qe, qs, qb))
    nleg = min(199, 2 * top)
    mu, wt = np.polynomial.legendre.leggauss((nleg + 2 * top + 2) // 2)
    pi_, tau = np.zeros((2, k + 1, len(mu)))
    pin, pim = np.ones_like(mu), np.zeros_like(mu)
    for i in range(1, min(k, top) + 1):
        cn = (2 * i + 1) / (i * (i + 1.0))
        pi_[i], tau[i] = cn * pin, cn * (i * mu * pin - (i + 1) * pim)
        pin, pim = ((2 * i + 1) * mu * pin - (i + 1) * pim) / i, pin
    s1 = np.einsum("kzb,kq->zbq", a, pi_) + np.einsum("kzb,kq->zbq", b, tau)
    s2 = np.einsum("kzb,kq->zbq", b, pi_) + np.einsum("kzb,kq->zbq", a, tau)
    i1, i2 = abs(s1) ** 2, abs(s2) ** 2
    ph = [np.einsum("zbq,zb->zq", v, n) for v in (0.5 * (i2 + i1), 0.5 * (i2 - i1), (s2 * s1.conj()).real)]
    leg = np.polynomial.legendre.legvander(mu, nleg)
    coef = np.stack([(v * wt * (wl * wl / (np.pi * sca))[:, None]) @ leg for v in ph], 1) * (np.arange(nleg + 1) + 0.5)
    return ext, sca, back, coef


def _lobatto(n):
    """Positive nodes (ascending) and weights of the 2n-point Lobatto rule."""
    leg = np.polynomial.legendre.Legendre.basis(2 * n - 1)
    x = leg.deriv().roots().real
    for _ in range(3):
        x = x - leg.deriv()(x) / leg.deriv(2)(x)
    mu = np.append(np.sort(x[x > 1e-9]), 1.0)
    return mu, 2.0 / ((2 * n) * (2 * n - 1) * leg(mu) ** 2)


def _phase(coef, mu):
    """Azimuthal mean of the (I, Q) phase matrix for scattering from +mu and
    from -mu into +mu: [2][n][n], rows outgoing."""
    nleg, N = coef.shape[1] - 1, len(mu)
    npts = 2 * ((nleg + 1) // 2) + 4
    phi = 2 * np.pi * np.arange(npts) / npts
    out = np.zeros((2, 2 * N, 2 * N))
    for q, sg in enumerate((1.0, -1.0)):
        m1, m2 = sg * mu[None, :, None], mu[:, None, None]
        t1, t2 = np.sqrt(1 - m1 * m1), np.sqrt(1 - m2 * m2)
        cs = m1 * m2 + t1 * t2 * np.cos(phi)
        v = [np.polynomial.legendre.legval(np.clip(cs, -1, 1), c) for c in coef]
        ss = np.sqrt(np.maximum(0.0, 1 - cs * cs))
        ok = ss > 1e-9
        r = 1.0 / np.where(ok, ss, 1.0)
        sin1, sin2 = np.where(ok, t2 * np.sin(phi) * r, 0.0), np.where(ok, t1 * np.sin(phi) * r, 0.0)
        cos1 = np.where(ok, (t1 * m2 - t2 * m1 * np.cos(phi)) * r, 1.0)
        cos2 = np.where(ok, (t2 * m1 - t1 * m2 * np.cos(phi)) * r, -1.0)
        c1, c2, s1, s2 = 1 - 2 * sin1 ** 2, 1 - 2 * sin2 ** 2, 2 * sin1 * cos1, 2 * sin2 * cos2
        out[q, 0::2, 0::2] = v[0].mean(-1)
        out[q, 0::2, 1::2] = (v[1] * c1).mean(-1)
        out[q, 1::2, 0::2] = (v[1] * c2).mean(-1)
        out[q, 1::2, 1::2] = (v[0] * c1 * c2 - v[2] * s1 * s2).mean(-1)
    return out


def _planck(t, wl):
    return 1.1911e8 / wl ** 5 / (np.exp(1.4388e4 / (wl * t)) - 1)


def _scattering_layer(ph, ext, emis, gas, dz, b0, b1, mu, w):
    """R, T and the sources S+, S- of a layer by doubling."""
    nd = max(0, int(math.log(max((ext + gas) * dz, 1e-7) / 1e-6) / math.log(2.0)) + 1)
    n = 2 * len(mu)
    m2, w2 = np.repeat(mu, 2), np.repeat(w, 2)
    step = dz / 2.0 ** nd / m2[:, None]
    R = 2 * np.pi * step * w2 * ph[1]
    T = np.eye(n) - step * ((ext + gas) * np.eye(n) - 2 * np.pi * w2 * ph[0])
    src = np.where(np.arange(n) % 2 == 0, b0 * step[:, 0] * (emis + gas), 0.0)
    sp, sm, cp, cm = src, src, src, src
    fac = (b1 / b0 - 1.0) / 2.0 ** nd
    for _ in range(nd):
        W = T @ np.linalg.inv(np.eye(n) - R @ R)
        low = sm + fac * cm
        sp, sm, cp, cm = (sp + W @ (sp + R @ low) + fac * cp, sm + W @ (low + R @ sp), cp + W @ (cp + R @ cm),
                          cm + W @ (cm + R @ cp))
        R, T = R + W @ R @ T, W @ T
        fac = 2 * fac
    return R, R, T, T, sp, sm


def _clear_layer(gas, dz, b0, b1, mu):
    path = np.repeat(dz * gas / mu, 2)
    e, slope = np.exp(-path), (b1 - b0) / path
    on = np.arange(len(path)) % 2 == 0
    sp = np.where(on, b1 - slope - (b1 - slope * (1 + path)) * e, 0.0)
    sm = np.where(on, b0 + slope - (b0 + slope * (1 + path)) * e, 0.0)
    z = np.zeros((len(path),) * 2)
    return z, z, np.diag(e), np.diag(e), sp, sm


def _combine(u, v):
    (rp1, rm1, tp1, tm1, sp1, sm1), (rp2, rm2, tp2, tm2, sp2, sm2) = u, v
    i = np.eye(len(sp1))
    gp, gm = np.linalg.inv(i - rp1 @ rm2), np.linalg.inv(i - rm2 @ rp1)
    return (rp2 + tp2 @ gp @ rp1 @ tm2, rm1 + tm1 @ gm @ rm2 @ tp1, tp2 @ gp @ tp1, tm1 @ gm @ tm2,
            sp2 + tp2 @ (gp @ (sp1 + rp1 @ sm2)), sm1 + tm1 @ (gm @ (sm2 + rm2 @ sp1)))


def _radiance(up, dn, sky, gnd):
    rp, _, tp, _, sp, _ = up
    _, rm, _, tm, _, sm = dn
    i = np.eye(len(sky))
    down = np.linalg.solve(i - rp @ rm, rp @ (tm @ gnd) + tp @ sky + rp @ sm + sp)
    return np.linalg.solve(i - rm @ rp, rm @ (tp @ sky) + tm @ gnd + rm @ sp + sm), down


def _tb(rad, wl):
    i, q = rad[0::2], rad[1::2]
    return 1.4388e4 / (wl * np.log(1.0 + 1.1911e8 / (np.stack([i + q, i - q], -1) * wl ** 5)))


def _column(p, c, freqs, N, emissivity):
    """tb [2 levels][2N][F][2], Ze, hydrometeor and gas attenuation [F][L]."""
    hl, tl, pl, rl = (np.asarray(p[k]).reshape(-1, p["max_nlyrs"] + 1)[c] for k in ("hgt_lev", "temp_lev", "press_lev",
                                                                                  "relhum_lev"))
    L, dz = len(hl) - 1, np.diff(hl)
    t, rh, pr = 0.5 * (tl[1:] + tl[:-1]), 0.5 * (rl[1:] + rl[:-1]), np.sqrt(pl[1:] * pl[:-1])
    x = 373.16 / t
    es = 1013.246 * 10 ** (-7.90298 * (x - 1) + 5.02808 * np.log10(x) - 1.3816e-7 * (10 ** (11.344 * (1 - 1 / x)) - 1) +
                           8.1328e-3 * (10 ** (-3.49149 * (x - 1)) - 1))
    e = rh * es
    qv = _RV / _RD * e / (pr - (1 - _RV / _RD) * e)
    q = np.asarray(p["hydro_q"]).reshape(-1, L, 2)[c]
    q = q * (pr / (_RD * (1 + (_RV / _RD - 1) * qv - q.sum(1)) * t))[:, None]
    wet = np.nonzero(q.sum(1) > 0)[0]
    mu, w = _lobatto(N)
    tb = np.zeros((2, 2 * N, len(freqs), 2))
    ze, ah, aa = np.full((len(freqs), L), -9999.0), np.zeros((len(freqs), L)), np.zeros((len(freqs), L))
    for k, f in enumerate(freqs):
        wl = _C / (f * 1e3)
        gas, m = _gas(f, t, e / (t * _RV), pr), _water(t[wet], f)
        sp = [_mie(f, d, n, m) for d, _, n in (_bins(row, q[wet, h]) for h, row in
                                              enumerate((workloads.CLOUD_C1, workloads.RAIN_C1)))]
        layers = {}
        for j, z in enumerate(wet):
            nleg, coef = 0, np.zeros((3, 400))
            for _, sca, _, cf in sp:
                nleg = max(nleg, int(np.nonzero(cf[j, 0] > 1e-7)[0][-1]))
                top = min(nleg, cf.shape[2])
                coef[:, :top] += cf[j, :, :top] * sca[j]
            ext, sca = sum(s[0][j] for s in sp), sum(s[1][j] for s in sp)
            ph = _phase(coef[:, :nleg + 1] / (4 * np.pi), mu)
            layers[z] = _scattering_layer(ph, ext, ext - sca, gas[z], dz[z], _planck(tl[z + 1], wl), _planck(tl[z], wl), mu, w)
            back = sum(s[2][j] for s in sp)
            ze[k, z] = 10 * math.log10(1e18 / (0.93 * np.pi ** 5) * back * (wl * 1e-6) ** 4)
            ah[k, z] = 10 * math.log10(math.exp(ext * dz[z]))
        aa[k] = 10 * np.log10(np.exp(gas * dz))
        stack = None
        for z in range(L - 1, -1, -1):
            lay = layers.get(z) or _clear_layer(gas[z], dz[z], _planck(tl[z + 1], wl), _planck(tl[z], wl), mu)
            stack = lay if stack is None else _combine(stack, lay)
        zero, one, none = np.zeros((2 * N, 2 * N)), np.eye(2 * N), np.zeros(2 * N)
        even = np.arange(2 * N) % 2 == 0
        sfc = (zero, (1 - emissivity) * one, one, one, none, none)
        gnd, sky = np.where(even, emissivity * _planck(290.0, wl), 0.0), np.where(even, _planck(2.73, wl), 0.0)
        top, low = (zero, zero, one, one, none, none), _combine(stack, sfc)
        for lev, (a, b) in enumerate(((top, low), (stack, sfc))):
            up, dn = _radiance(a, b, sky, gnd)
            tb[lev, N - 1::-1, k], tb[lev, N:, k] = _tb(up, wl), _tb(dn, wl)
    return tb, ze, ah, aa


def exact(case, seed):
    """The outputs of the cloud and rain cases with up to EXACT_COLUMNS columns
    from plain numpy.  None for more columns (minutes), for the split form's
    larger batches and for the T-matrix (its solve needs more than 64 bits to
    be a reference)."""
    if case["entry"] == "tmatrix" or case.get("kind", "cloud_rain") != "cloud_rain":
        return None
    if case["cols"] > EXACT_COLUMNS or case["layers"] * case["freqs"] > 400:
        return None
    pam, N, freqs = _cloud_rain(case, seed), case.get("nummu", 16), _channels(case["freqs"])
    cols = [_column(pam.p, c, freqs, N, 0.5) for c in range(case["cols"])]
    tb = np.stack([c[0] for c in cols])
    ang = np.degrees(np.arccos(_lobatto(N)[0]))
    ang = np.concatenate([180.0 - ang[::-1], ang])
    n, F = len(cols), len(freqs)
    if case["entry"] == "profile":
        return dict(tb=tb[:, None], emissivity=np.full((n, 1, 2, F, N), 0.5), angles_deg=ang, status=None,
                    Ze=np.stack([c[1].T for c in cols])[:, None, :, :, None, None],
                    Att_hydro=np.stack([c[2].T for c in cols])[:, None, :, :, None],
                    Att_atmo=np.stack([c[3].T for c in cols])[:, None])
    return dict(tb=tb, emissivity=np.full((n, 2, F, N), 0.5), angles_deg=ang, status=None)
