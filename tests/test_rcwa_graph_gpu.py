"""What a cached graph of celeris_rcwa_batch holds: a batch of a shape seen before, with another
symmetry tolerance, does not replay the old one's graph; its kernels are counted; and the
buckets of a batch (cells of one size and path) run beside one another.
"""
import os
import time

import numpy as np
import pytest

from celeris_b200 import capi

pytestmark = pytest.mark.gpu

BASE = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=4.0, eps_bg=1.0, thickness_um=0.6)


def launches(cells):
    """Kernels that one batch launches, once its shape is known (tuned and captured)."""
    arr = [capi.rcwa_cell(**c) for c in cells]
    lib = capi.load()
    for _ in range(2):
        before = lib.celeris_launch_count()
        res, info = capi.rcwa_batch(arr)
        assert not info.any()
    return lib.celeris_launch_count() - before, res


@pytest.mark.parametrize("grid", [0, 64])
def test_symmetry_tolerance_of_a_known_shape(grid):
    """Tolerance 0 sends every cell to the order basis: more kernels, the same results. The
    default and 0 agree in their first six decimals."""
    cells = [dict(BASE, Mx=2, fill_x=0.3 + 0.1 * i, shape=1 if grid else 0, grid=grid) for i in range(5)]
    count, res = launches(cells)
    os.environ["CELERIS_RCWA_SYM_TOL"] = "0"
    try:
        redo, res0 = launches(cells)
    finally:
        del os.environ["CELERIS_RCWA_SYM_TOL"]
    assert redo > count
    assert launches(cells)[0] == count
    for a, b in zip(res, res0):
        assert abs(a["tx0"] - b["tx0"]) <= 1e-10 and abs(a["R"] - b["R"]) <= 1e-10


@pytest.mark.parametrize("extra,kernels", [
    (dict(), 4),  # class operators, two-port, expansion, outputs
    (dict(shape=1, grid=64), 5),  # and the phase table
    (dict(theta_rad=0.2), 3),  # operators, two-port, outputs
    (dict(theta_rad=0.2, shape=1, grid=64), 5),  # two phase tables
    (dict(thickness_um=5e-4), 7),  # class operators, three eigen stages, class S-matrix, expansion, outputs
    (dict(thickness_um=5e-4, shape=1, grid=64), 8),
    (dict(thickness_um=5e-4, theta_rad=0.2), 8),  # operators, M, three eigen stages, two S-matrix stages, outputs
    (dict(thickness_um=5e-4, theta_rad=0.2, shape=1, grid=64), 10),
])
def test_launch_count_of_a_bucket(extra, kernels):
    assert launches([dict(BASE, Mx=2, fill_x=0.5, **extra)])[0] == kernels


def test_buckets_run_side_by_side():
    """Twenty thin M = 4 cells (eigendecomposition, ~1.5 ms) and twenty M = 5 cells (two-port,
    ~0.8 ms) leave most of the chip idle alone: together they take less than one after the other."""
    def median_time(cells):
        arr, t = [capi.rcwa_cell(**c) for c in cells], []
        for _ in range(15):
            t0 = time.perf_counter()
            capi.rcwa_batch(arr)
            t.append(time.perf_counter() - t0)
        return float(np.median(t[3:]))

    thin = [dict(BASE, Mx=4, fill_x=0.2 + 0.03 * i, thickness_um=2e-3) for i in range(20)]
    thick = [dict(BASE, Mx=5, fill_x=0.2 + 0.03 * i) for i in range(20)]
    a, b, both = (median_time(c) for c in (thin, thick, thin + thick))
    assert both <= 0.85 * (a + b), (a, b, both)
