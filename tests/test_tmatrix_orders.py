"""T-matrix kernels over the orders and batches where their routes change.

A particle's solves go side by side or one by one by its order: steps of the
convergence search share the CTA up to NMAX 35, the m >= 1 solves up to about
22; records of the amplitude kernel beyond 1 GB take several rounds.  Each
size runs upright and canted, next to an empty bin, against the REAL*16
oracle.  Tolerance: 2e-6 of an array's largest magnitude, as for all
T-matrix outputs (T rounded to single precision by both sides; the FP64 solve
adds less than 1e-9 at these sizes and aspect ratios).
"""
import numpy as np
import pytest
from test_tmatrix import C, _compare, _item, _oracle_item, _run_gpu

FREQ = 89e9


def _ice(x, asr, canting):
    """Solid-ice bins of equal-volume size parameters x; the last one empty."""
    d = [2.0 * xi * C / (2.0 * np.pi * FREQ) / (asr ** (1.0 / 3.0) if asr <= 1.0 else asr ** (-2.0 / 3.0)) for xi in x]
    return _item(FREQ, 1.78 - 0.003j, -1, d + [d[0]], [1e3] * len(x) + [0.0], 917.0, asr, canting)


@pytest.mark.gpu
@pytest.mark.parametrize("x, asr, nummu", [
    ((0.02, 0.3), 0.8, 32),    # NMAX 4 - 6
    ((4.0, 8.0), 0.6, 16),     # all orders side by side
    ((9.5, 11.0), 0.6, 8),     # around the last such NMAX
    ((15.0, 20.0), 1.0, 8),    # search side by side, m >= 1 one by one
    ((22.0, 25.0), 1.0, 8),    # around the end of the side-by-side search
])
def test_gpu_tmatrix_orders(oracle_mod, x, asr, nummu):
    items = [_ice(x, asr, 0.0), _ice(x, asr, 30.0)]
    out = _run_gpu(items, len(x) + 1, nummu)
    _compare(out, [_oracle_item(oracle_mod, it, nummu) for it in items], nummu)
    assert np.all(out["nmax"][:, :-1] > 0) and np.all(out["nmax"][:, -1] == 0)
    assert np.array_equal(out["nmax"][0], out["nmax"][1])


@pytest.mark.gpu
@pytest.mark.parametrize("node", [0, 4, 7])
def test_gpu_tmatrix_axis_along_an_angle(oracle_mod, node):
    """A canted particle whose axis is one of the incident directions (a Lobatto
    node, the last one 0 deg): the particle frame's azimuth is singular there."""
    leg = np.polynomial.legendre.Legendre.basis(15).deriv().roots()  # Gauss-Lobatto rule of 16 points
    mu = np.append(np.sort(leg[leg > 0]), 1.0)[node]
    beta = float(np.degrees(np.arccos(mu)))
    items = [_ice((0.5, 2.0), 0.6, b) for b in (beta, 180.0 - beta)]
    out = _run_gpu(items, 3, 8)
    _compare(out, [_oracle_item(oracle_mod, it, 8) for it in items], 8)


@pytest.mark.gpu
def test_gpu_tmatrix_record_rounds(oracle_mod):
    """More particles than one round of records holds (about 2800 of each kind
    here), upright and canted in turn, some invalid: equal particles give
    equal bytes, whichever round they are in."""
    n, nummu = 7000, 32
    kinds = [_item(FREQ, 1.78 - 0.003j, -1, [2.0e-3], [1e3], 917.0, 0.6, canting) for canting in (0.0, 30.0)]
    bad = _item(FREQ, 1.78 - 0.003j, -1, [2.0e-3], [1e3], 917.0, -1.0, 0.0)
    items = [bad if i % 1000 == 999 else kinds[i % 2] for i in range(n)]
    out = _run_gpu(items, 1, nummu)
    _compare(out, [_oracle_item(oracle_mod, it, nummu) for it in kinds], nummu)
    good = np.array([i % 1000 != 999 for i in range(n)])
    assert np.all((out["status"] == 0) == good)
    for k in ("scatter_matrix", "extinct_matrix", "emis_vector", "sback", "back_spec", "nmax"):
        v = np.asarray(out[k]).reshape(n, -1)
        for c in (0, 1):
            sel = good & (np.arange(n) % 2 == c)
            assert np.all(v[sel] == v[c]), (k, c)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1e-80, 1e-120])
def test_gpu_tmatrix_vanishing_pivots(oracle_mod, d):
    """Particles so small that the Bessel functions overflow: every system of all
    steps of the side-by-side search loses its pivots at once.  The bins say
    FATAL | ST_RANGE, and the bins beside them keep their bytes."""
    fine = _ice((0.3, 2.0), 0.8, 0.0)
    mixed = {k: (v[:1] + [w] * 4 + v[1:] if isinstance(v, list) else v)
             for k, v, w in ((k, fine[k], fine[k][0] if isinstance(fine[k], list) else None) for k in fine)}
    mixed["dmax"][1:5] = [d] * 4
    want = _run_gpu([fine], 3, 8)
    out = _run_gpu([mixed], 7, 8)
    assert int(out["status"][0]) == (2 | 0x10000)
    assert np.all(out["nmax"][0, 1:5] < 0)
    for k in ("scatter_matrix", "extinct_matrix", "emis_vector", "sback"):
        assert np.array_equal(out[k][0], want[k][0]), k
    assert np.array_equal(np.delete(out["back_spec"][0], range(1, 5)), want["back_spec"][0])
