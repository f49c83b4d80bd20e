"""Full spectra with a bin whose diameter has no Mie series (NaN, negative) or
one too long for it: the column's status says FATAL | ST_SIZE, and the other
columns keep the bytes they have without that bin.  The bin stands first,
between and last of its 40, in a lane of its own pass; an empty bin with such a
diameter takes no part except as the last one, which sizes the series."""
import numpy as np
import pytest

from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu
FREQS = [23.8, 150.0]


def _run(pam):
    pam.runPamtra(FREQS, failOnError=False)
    return {k: np.array(pam.r[k])[:, 0] for k in ("status", "tb", "kexttot_all", "salbedo_all")}


@pytest.mark.parametrize("species", [0, 1])
@pytest.mark.parametrize("at", [0, 17, 39])
@pytest.mark.parametrize("value", [np.nan, -3e-4, 1.0, np.inf])
def test_bin_without_a_series(native, species, at, value):
    pam = wl.fullspec_pam(ncol=3, nlay=6, seed=5)
    pam.nmlSet["save_ssp"] = True
    good = _run(pam)
    assert not good["status"].any()
    fs = pam.df.dataFullSpec
    z = int(np.argmax(fs["n_ds"][1, 0, :, species, 17] > 0))
    fs["d_ds"][1, 0, z, species, at] = value
    bad = _run(pam)
    assert np.all(bad["status"][1] & (2 | native.ST_SIZE) == (2 | native.ST_SIZE))
    for k, v in bad.items():
        assert np.array_equal(v[[0, 2]], good[k][[0, 2]]), k
    fs["n_ds"][1, 0, z, species, at] = 0.0
    empty = _run(pam)
    assert np.all(empty["status"][1] == 0) == (at != 39)
