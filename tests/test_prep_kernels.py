"""Column preparation on the GPU where its warps have remainders: bin counts
around the warp width and at the limit of 256, fixed and adaptive grids,
against the oracle; batches around the 32 columns of one compaction block,
with empty columns, against the columns run one by one.

Tolerances: a log-grid boundary is exp(w i + log d_1) with |log d_1| <= 17,
so three roundings and a last-bit difference of log and exp between the two
libraries move it by at most about 2e-14 relative; bounds of 1e-13 on
diameters.  A bin width is a difference of two boundaries (1e-13 d absolute),
and the number in a bin adds lambda d <= 60 times that in the exponent.
"""
import copy

import numpy as np
import pytest

from pamtra_b200 import batch as pbatch
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("nbin", [1, 2, 31, 32, 33, 64, 255, 256])
def test_psd_bins_match_oracle(oracle_mod, native, nbin, adaptive):
    pam = wl.golden_pam()
    for row in range(2):
        pam.df.data["nbin"][row] = nbin
    pam.nmlSet["hydro_adaptive_grid"] = adaptive
    pam.nmlSet["save_psd"] = True
    ref, err = oracle_mod.run_pamtra(copy.deepcopy(pam), [10.65])
    pam.runPamtra([10.65], failOnError=False)
    assert (pam.fortError == 0) == (err == 0)
    if err:
        return
    d, dd, n = ref["psd_d"], ref["psd_deltad"], ref["psd_n"]
    assert np.array_equal(pam.r["psd_d"] == -9999, d == -9999)
    on = d != -9999
    np.testing.assert_allclose(pam.r["psd_d"][on], d[on], rtol=1e-13)
    np.testing.assert_allclose(pam.r["psd_mass"][on], ref["psd_mass"][on], rtol=4e-13)
    assert np.all(np.abs(pam.r["psd_deltad"] - dd)[on] <= 1e-13 * d[on])
    assert np.all(np.abs(pam.r["psd_n"] - n)[on] <= np.abs(n[on]) * (1e-11 + 2e-13 * d[on] / dd[on]))


@pytest.mark.parametrize("ncol", [31, 32, 33, 70])
def test_compaction_of_ragged_batch(native, ncol):
    b = wl.uneven_batch(ncol, seed=50 + ncol, nummu_choices=(8,), nfreq_range=(1, 2))
    q = b.host["hydro_q"]
    q[[0, 5, 17, ncol - 1]] = 0.0           # columns without hydrometeors, the first and the last among them
    q[3, 33:] = 0.0
    b = pbatch.pack_columns(b.settings, b.species, b.host, b.species_stride)
    tb = pbatch.run(b, 0)["tb"].cpu().numpy()
    status = pbatch.run(b, 0)["status"].cpu().numpy()
    assert not status.any()
    for c in (0, 1, 3, 4, 17, 30, ncol - 2, ncol - 1):
        one = pbatch.subset(b, [c])
        t1 = pbatch.run(one, 0)["tb"].cpu().numpy()
        assert np.array_equal(t1[0], tb[c][:, :, :t1.shape[3]])
