"""Columns whose number of layers is refused (below 2 or above max_nlyrs): their
status says FATAL | ST_SIZE and tb stays -9999, and every other column of the
batch keeps the bytes it has without them, in each form and NUMMU.  The refused
columns carry enough scattering layers for several segments of the adding,
and stand first, between and last, where a count that runs past the column's
rows meets a neighbour's or the end of the arrays."""
import numpy as np
import pytest

from pamtra_b200 import batch as pbatch
from pamtra_b200 import packing
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _run(b, prec, dev):
    import torch
    out = b.alloc_outputs(dev, ssp=True)
    shape = out["kexttot"].shape
    for k in ("ze", "att_hydro", "att_atmo"):
        out[k] = torch.zeros(shape, dtype=torch.float64, device=dev)
    pbatch.run(b, 0, out, precision=prec)
    torch.cuda.synchronize()
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("nummu", [8, 16, 32])
@pytest.mark.parametrize("refused", [(0, 3, 7), (0, 1, 7)])
def test_refused_columns_leave_the_others_alone(native, nummu, refused):
    import torch
    dev = torch.device("cuda", 0)
    b = wl.uneven_batch(8, seed=90 + nummu, nummu_choices=(nummu,), nfreq_range=(2, 3))
    h = b.host
    lm = int(h["max_nlyrs"])
    q = h["hydro_q"].reshape(8, lm, -1)
    for c in refused:  # twelve scattering layers at the bottom, whatever the column's species
        kinds = b.species.reshape(8, -1)[c]["dist"] != packing.DIST_CODES["disabled"]
        q[c, :12, int(np.argmax(kinds))] = 2e-4
    b.settings.active = 1
    nly = np.array(h["nlyrs"])
    for prec in (native.PREC_FP64, native.PREC_FP64_BATCHED, native.PREC_3XTF32, native.PREC_3XTF32_FP64ADD):
        good = _run(pbatch.pack_columns(b.settings, b.species, dict(h, nlyrs=nly), b.species_stride), prec, dev)
        for counts in ((lm + 10, lm + 1, lm + 150), (1, 0, -3)):
            bad = nly.copy()
            bad[list(refused)] = counts
            got = _run(pbatch.pack_columns(b.settings, b.species, dict(h, nlyrs=bad), b.species_stride), prec, dev)
            for c in range(8):
                nf = int(h["nfreq"][c])
                if c in refused:
                    assert np.all(got["status"][c, :nf] == (2 | native.ST_SIZE)), (prec, c)
                    assert np.all(got["tb"][c] == -9999.0)
                    assert np.all(got["num_doubles"][c] == -1) and np.all(got["kexttot"][c] == 0.0)
                    assert np.array_equal(got["emissivity"][c], good["emissivity"][c])
                    continue
                assert np.array_equal(got["tb"][c], good["tb"][c]), (prec, c)
                for k in ("status", "kextatmo", "kexttot", "salbedo", "num_doubles", "ze", "att_hydro", "att_atmo"):
                    assert np.array_equal(got[k][c, :nf], good[k][c, :nf], equal_nan=True), (prec, k, c)


def test_outputs_past_a_columns_frequencies(native):
    """Columns of fewer frequencies than the batch's widest: the per-layer outputs
    past them say that there is no layer (0, 0, -1), whatever the scratch held."""
    import torch
    dev = torch.device("cuda", 0)
    eng = native.Engine(0)
    for seed, nfr in ((70, (6, 6)), (71, (1, 6))):  # the first batch leaves its items in the scratch
        b = wl.uneven_batch(6, seed=seed, nummu_choices=(8,), nfreq_range=nfr)
        out = b.alloc_outputs(dev, ssp=True)
        pbatch.run(b, 0, out, eng=eng)
        torch.cuda.synchronize()
    out = {k: v.cpu().numpy() for k, v in out.items()}
    eng.close()
    past = np.arange(out["status"].shape[1])[None, :] >= b.host["nfreq"][:, None]
    assert past.any() and (out["num_doubles"][~past] >= 0).any()
    for k, v in (("kexttot", 0.0), ("salbedo", 0.0), ("num_doubles", -1)):
        assert np.all(out[k][past] == v), k
