"""The two FP64 forms run the same kernels: equal bytes, and the oracle (the
reference's order of operations, COMBINE_LAYERS4 layer by layer with two
inverses) within 1e-6 K on an uneven batch, for two columns of each NUMMU and
surface (specular, Lambertian).  This is the check of the adding's own order
(segments, reciprocity, one inverse), which no run of one form against the
other gives."""
import numpy as np
import pytest
from test_gpu_parity import TB_TOL, _oracle_packed_column, _run_prec

from pamtra_b200 import batch as pbatch
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def test_uneven_batch_of_both_forms(oracle_mod, native):
    b = wl.uneven_batch(24, seed=43, nfreq_range=(2, 3))
    h = b.host
    h["sfc_refl"] = np.where(np.arange(24) % 2, ord("L"), ord("S")).astype(np.int8)
    b.settings.emissivity = 0.6
    b = pbatch.pack_columns(b.settings, b.species, h, b.species_stride)
    plain = _run_prec(b, native.PREC_FP64)
    batched = _run_prec(b, native.PREC_FP64_BATCHED)
    for k in ("tb", "status"):
        assert np.array_equal(plain[k], batched[k]), k
    assert not plain["status"].any()
    for nummu in (8, 16, 32):
        for refl in b"SL":
            cols = np.nonzero((h["nummu"] == nummu) & (h["sfc_refl"] == refl))[0][:2]
            assert len(cols) == 2, (nummu, refl)
            for c in cols:
                err, t, n, nf = _oracle_packed_column(oracle_mod, b, int(c))
                assert err == 0 and n == nummu
                assert np.max(np.abs(plain["tb"][c][:, :2 * n, :nf, :] - t)) < TB_TOL, (nummu, chr(refl), c)
