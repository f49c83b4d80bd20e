"""run_host around the size where its inputs and outputs stop going through
one pinned copy each: the bytes of the device run, for batches below, across
(inputs above, outputs below) and beyond it, and for a small call after a large one."""
import numpy as np
import pytest

from pamtra_b200 import batch as pbatch
from pamtra_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1,), (33, 8), (90, 1, 90), (150, 33)])
def test_run_host_matches_device_run(native, sizes):
    for ncol in sizes:
        b = pbatch.pack_pam(wl.c2_pam(ncol, seed=5), [24.0, 89.0])
        host = pbatch.run_host(b, 0)
        dev = pbatch.run(b, 0)
        for k, v in dev.items():
            if hasattr(v, "cpu"):
                assert np.array_equal(np.asarray(host[k]), v.cpu().numpy(), equal_nan=True), (ncol, k)
