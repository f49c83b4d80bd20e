"""Adding in segments (k_adding): columns whose numbers of scattering layers
lie around the segment rule's steps (one segment up to 7, then about
sqrt(M) layers each), with clear layers on top, between and below, against the
oracle within 1e-6 K for each NUMMU and both surfaces, and the unscaled form that
takes the split-precision doubling's layers within the 0.05 K of that doubling.
"""
import warnings

import numpy as np
import pytest

import pamtra_b200 as pb
from pamtra_b200 import batch as pbatch
from pamtra_b200 import workloads as wl

FREQS = [23.8, 150.0]
COUNTS = (0, 1, 2, 7, 8, 9, 10, 16, 17, 25, 26, 37)


def segments(m):
    """Lengths of the segments of a unit with m scattering layers (the kernel's rule)."""
    if m < 8:
        return [m]
    ln = 4
    while ln * ln < m:
        ln += 1
    ns = (m + ln - 1) // ln
    return [m * (s + 1) // ns - m * s // ns for s in range(ns)]


def test_segments_hold_two_layer_records():
    for m in range(8, 2000):
        s = segments(m)
        assert sum(s) == m and min(s) >= 2 and max(s) <= max(4, int(np.ceil(np.sqrt(m))))


def _pam(m, refl):
    warnings.simplefilter("ignore")
    rng = np.random.default_rng(m)
    nlay = 40
    pam = pb.pyPamtra()
    pam.df.addHydrometeor(wl.CLOUD_C1)
    pam.df.addHydrometeor(wl.RAIN_C1)
    pam.nmlSet["hydro_adaptive_grid"] = False
    pam.nmlSet["emissivity"] = 0.6
    hl = np.linspace(0.0, 10000.0, nlay + 1)
    _, p, t = pb.meteoSI.usStandard(hl)
    q = np.zeros((nlay, 2))
    at = np.sort(rng.choice(nlay, m, replace=False))
    q[at, 1] = 10 ** rng.uniform(-4.5, -2.7, m)
    q[at[::2], 0] = 3e-4
    pam.createProfile(hgt_lev=hl, temp_lev=t, press_lev=p, relhum_lev=np.full(nlay + 1, 70.0), hydro_q=q,
                      sfc_refl=refl, obs_height=np.tile([833000.0, 0.0], (1, 1, 1)))
    return pam


def _oracle(oracle_mod, refl, nummu):
    out = []
    for m in COUNTS:
        r, err = oracle_mod.run_pamtra(_pam(m, refl), FREQS, nummu=nummu)
        assert err == 0
        out.append(r["tb"][0, 0])
    return np.stack(out)


@pytest.mark.gpu
@pytest.mark.parametrize("refl", ["S", "L"])
@pytest.mark.parametrize("nummu", [8, 16, 32])
def test_segment_counts_match_oracle(oracle_mod, native, nummu, refl):
    b, _ = pbatch.concat([pbatch.pack_pam(_pam(m, refl), FREQS, nummu=nummu) for m in COUNTS])
    ref = _oracle(oracle_mod, refl, nummu)
    bounds = {native.PREC_FP64: 1e-6, native.PREC_FP64_BATCHED: 1e-6, native.PREC_3XTF32_FP64ADD: 0.05,
              native.PREC_3XTF32: 0.05}
    for prec, tol in bounds.items():
        out = pbatch.run(b, 0, precision=prec)
        assert not out["status"].cpu().numpy().any()
        tb = out["tb"].cpu().numpy()
        assert np.max(np.abs(tb - ref)) < tol, prec
        again = pbatch.run(b, 0, precision=prec)["tb"].cpu().numpy()
        assert np.array_equal(tb, again)
