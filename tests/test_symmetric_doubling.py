"""FP64 doubling in the scaled symmetric form (k_layer): columns whose layers
walk every branch of the inverse -- G = I + X for thin layers, further terms,
squarings, elimination -- for each NUMMU, against the oracle within 1e-6 K.

``branches`` follows the kernel's choice on the CPU: the phase matrices come
from the oracle, the doubling is plain numpy, and the norm of X = R R is its
trace in the scaled form (the row-sum norm too above 0.5).  The scaled R of
the oracle's phase matrices is symmetric to rounding, the property the
kernel rests on.
"""
import copy

import numpy as np
import pytest

from pamtra_b200 import workloads as wl

# graupel spheres (400 kg/m3, 0.1-6 mm, exponential with effective radius 1 mm): nearly conservative scattering
GRAUPEL = ("gwc_q", -99.0, -1, 400.0, -99.0, -99.0, -99.0, -99.0, 3, 40, "exp", -99.0, 1.0e-3, -99.0, -99.0,
           1.0e-4, 6.0e-3, "mie-sphere", "heymsfield10_particles", -99.0)
FREQS = [10.65, 89.0, 183.31]


def _pam():
    from pamtra_b200 import core, importer
    pam = core.pyPamtra()
    pam.df.addHydrometeor(wl.RAIN_GOLDEN)
    pam.df.addHydrometeor(GRAUPEL)
    pam.nmlSet["hydro_adaptive_grid"] = False
    pam = importer.createUsStandardProfile(pam, hgt_lev=[0.0, 400.0, 1000.0, 3000.0, 7000.0, 9000.0])
    pam.p["hydro_q"][0, 0, :, 0] = [1e-3, 1e-5, 0.0, 0.0, 0.0]
    pam.p["hydro_q"][0, 0, :, 1] = [0.0, 1e-6, 5e-4, 2e-3, 5e-2]
    return pam


def branches(oracle_mod, nummu):
    r, err = oracle_mod.run_pamtra(_pam(), FREQS, nummu=nummu, debug=True)
    assert err == 0
    d = r["debug"][0]
    mu, w = oracle_mod.lobatto(nummu)
    mu2, w2 = np.repeat(mu, 2), np.repeat(w, 2)
    s = np.sqrt(mu2 * w2)
    n = 2 * nummu
    hit = set()
    p = _pam().p
    dz = np.diff(p["hgt_lev"][0, 0])
    for f in range(len(FREQS)):
        for z in np.nonzero(d["present"])[0]:
            nd = int(d["num_doubles"][f, z])
            q = d["scatter_matrix"][f, z].reshape(4, n, n)
            step = dz[z] / 2.0 ** nd / mu2[:, None]
            ext = d["ext"][f, z] + max(d["kextatmo"][f, z], 0.0)
            R = 2 * np.pi * step * w2 * q[1]
            T = np.eye(n) - step * (ext * np.eye(n) - 2 * np.pi * w2 * q[0])
            Rs = s[:, None] * R / s
            assert np.max(np.abs(Rs - Rs.T)) <= 1e-12 * np.max(np.abs(Rs))
            for _ in range(nd):
                Rs = s[:, None] * R / s
                X = R @ R
                nrm = np.sum(Rs * Rs)
                if nrm > 0.5:
                    nrm = min(nrm, np.max(np.sum(np.abs(X), axis=1)))
                if nrm * nrm <= 5e-17:
                    hit.add("thin")
                else:
                    m, pw = 1, nrm
                    while pw > 5e-17 and m < 8:
                        pw, m = pw * pw, m + 1
                    kh, ph = 0, nrm * nrm
                    while ph > 5e-17 and kh < 2 * (m - 1):
                        ph, kh = ph * nrm, kh + 1
                    hit.add("elimination" if m >= 8 else "terms" if kh <= 7 * (m - 1) // 4 else "squarings")
                G = np.linalg.inv(np.eye(n) - X)
                R, T = R + T @ G @ R @ T, T @ G @ T
    return hit


@pytest.mark.parametrize("nummu", [8, 16, 32])
def test_columns_walk_every_branch(oracle_mod, nummu):
    assert branches(oracle_mod, nummu) == {"thin", "terms", "squarings", "elimination"}


@pytest.mark.gpu
@pytest.mark.parametrize("nummu", [8, 16, 32])
def test_every_branch_matches_oracle(oracle_mod, native, nummu):
    from pamtra_b200 import batch as pbatch
    ref, err = oracle_mod.run_pamtra(copy.deepcopy(_pam()), FREQS, nummu=nummu)
    assert err == 0
    b = pbatch.pack_pam(_pam(), FREQS, nummu=nummu)
    for prec in (native.PREC_FP64, native.PREC_FP64_BATCHED):
        out = pbatch.run(b, 0, precision=prec)
        assert not out["status"].cpu().numpy().any()
        assert np.max(np.abs(out["tb"].cpu().numpy() - ref["tb"].reshape(out["tb"].shape))) < 1e-6
