"""scatcnv weight tables of a context whose table could not be allocated at
first: that run takes the direct azimuth sums (within the 1e-6 K of all
FP64 brightness temperatures of the tables' one), and the next run, with memory
for the table, gives the bytes of a context that had it from the start.

The allocation fails because a tensor holds all but less than the table's size
(215 MB for NUMMU 32) of the device's memory; the kernels have run before, so
nothing else needs memory then."""
import numpy as np
import pytest

from pamtra_b200 import batch as pbatch
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def test_table_that_comes_late(native):
    import torch
    dev = torch.device("cuda", 0)
    b = wl.uneven_batch(3, seed=61, nummu_choices=(32,), nfreq_range=(2, 3))

    def run(eng):
        out = b.alloc_outputs(dev)
        pbatch.run(b, 0, out, eng=eng)
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in out.items()}

    first = native.Engine(0)
    want = run(first)
    assert not want["status"].any()
    late = native.Engine(0)
    late.reserve(late.workspace_bytes(b.columns(b.device_arrays(dev))))
    run_out = b.alloc_outputs(dev)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info(dev)[0]
    held = torch.empty(free - (128 << 20), dtype=torch.uint8, device=dev)
    try:
        assert torch.cuda.mem_get_info(dev)[0] < (200 << 20)
        pbatch.run(b, 0, run_out, eng=late)
        torch.cuda.synchronize()
    finally:
        del held
        torch.cuda.empty_cache()
    direct = run_out["tb"].cpu().numpy()
    assert not run_out["status"].cpu().numpy().any()
    assert np.max(np.abs(direct - want["tb"])) < 1e-6
    got = run(late)
    for k in ("status", "tb"):
        assert np.array_equal(got[k], want[k]), k
    late.close()
    first.close()
