"""Mie sums where the tiles of k_mie have remainders: bins around groups of
eight and passes of 32, series of about 5 to 60 terms (fours; 64 Legendre
orders per chunk; odd and even numbers of angle tiles; passes of fewer than 32
bins), against the oracle; and the two tile shapes against each other.
Tolerance: that of all single-scattering outputs, 1e-9 relative.
"""
import numpy as np
import pytest
import test_single_scattering_parity as ssp

from pamtra_b200 import batch as pbatch
from pamtra_b200 import packing
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu
FREQS = [5.0, 31.4, 53.0, 89.0, 157.0, 190.31, 243.0, 325.0, 448.0]


def _batch(nbins, nlay=5, seed=41):
    rng = np.random.default_rng(seed)
    kinds = ["rwc", "swc", "gwc", "iwc"]
    sp = np.empty(4, dtype=packing.SPECIES_DTYPE)
    for j, k in enumerate(kinds):
        sp[j] = wl._species_row(k, np.random.default_rng(300 + j), nbin=nbins[j], gamma=(k != "rwc"), rho=400.0)
    qs = [[10 ** rng.uniform(-4.0, -2.7) for _ in kinds]]
    b = wl._packed(wl._settings(16), sp, 0, np.array([nlay]), [FREQS], None, [kinds], qs, np.array([9000.0]), rng, nlay,
                   4, False)
    b.host["temp_lev"][0, :nlay + 1] = np.linspace(295.0, 245.0, nlay + 1)
    return b


@pytest.mark.parametrize("nbins", [(2, 7, 8, 9), (31, 32, 33, 40), (24, 25, 64, 65)])
def test_mie_tiles_match_oracle(oracle_mod, native, nbins):
    import torch
    dev = torch.device("cuda", 0)
    b = _batch(nbins)
    out = ssp._outputs(b, dev)
    pbatch.run(b, 0, out)
    torch.cuda.synchronize()
    assert ssp._compare(b, out, oracle_mod, 16) >= 9
    eng = native.engine(0)
    keep = eng.get_launch()
    try:
        eng.set_launch((2, 0, 0, 0, 8))
        two = ssp._outputs(b, dev)
        pbatch.run(b, 0, two)
        torch.cuda.synchronize()
    finally:
        eng.set_launch(keep)
    for k in ("kexttot", "salbedo", "scatter_matrix", "tb"):
        assert torch.equal(out[k], two[k]), k


@pytest.mark.parametrize("nummu", [8, 32])
def test_phase_matrices_of_even_and_odd_series(oracle_mod, native, nummu):
    """scatcnv from the pair table: the frequencies give species series of even
    and odd length; 36 and 528 angle pairs, one and three per thread.  A
    frequency whose phase function the angles do not resolve fails CHECK_NORM4
    on both sides."""
    import copy

    import torch
    dev = torch.device("cuda", 0)
    b = _batch((8, 8, 16, 8), nlay=3)
    st = copy.copy(wl._settings(nummu))
    passed = 0
    for f in FREQS:
        one = pbatch.pack_columns(st, b.species, dict(b.host, freqs=np.array([f]), max_nfreq=1),
                                  b.species_stride)
        out = ssp._outputs(one, dev)
        pbatch.run(one, 0, out)
        torch.cuda.synchronize()
        err = oracle_mod.run_column(oracle_mod.settings(st), one.species, one.host, 0, [f])[0]
        if err:
            assert int(out["status"][0, 0]) == (2 | native.ST_NORM)
            continue
        assert ssp._compare(one, out, oracle_mod, nummu) >= 1
        passed += 1
    assert passed >= 5


@pytest.mark.parametrize("nlay,nfreq", [(1, 1), (3, 1), (3, 3), (7, 9)])
def test_items_around_the_warps_of_a_cta(native, nlay, nfreq):
    """1, 3, 9 and 63 items in CTAs of 2, 4 and 8 warps: the last CTA is partly
    idle.  Items do not depend on one another, so the bytes are the same."""
    import torch
    b = _batch((8, 9, 16, 8), nlay=max(nlay, 2))
    q = b.host["hydro_q"]
    q[:, nlay:] = 0.0
    one = pbatch.pack_columns(b.settings, b.species, dict(b.host, freqs=np.array(FREQS[:nfreq]), max_nfreq=nfreq),
                              b.species_stride)
    eng = native.engine(0)
    keep = eng.get_launch()
    outs = []
    try:
        for warps in (2, 4, 8):
            eng.set_launch((warps, 0, 0, 0, 4))
            out = ssp._outputs(one, torch.device("cuda", 0))
            pbatch.run(one, 0, out)
            torch.cuda.synchronize()
            outs.append({k: out[k].clone() for k in ("kexttot", "salbedo", "scatter_matrix", "tb", "status")})
    finally:
        eng.set_launch(keep)
    assert int((outs[0]["kexttot"] > 0).sum()) == nlay * nfreq
    for o in outs[1:]:
        for k, v in o.items():
            assert np.array_equal(v.cpu().numpy(), outs[0][k].cpu().numpy(), equal_nan=True), (k, nlay, nfreq)
