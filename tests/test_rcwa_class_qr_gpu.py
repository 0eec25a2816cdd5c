"""Mirror-symmetric cells whose layer the two-port leaves to the eigendecomposition (thinner
than k0 h = 0.01 or of more than 100 rad of optical phase), solved in their parity classes,
against the oracle at the RCWA tests' parity tolerance. The thick layers absorb a little, so that
no resonance amplifies the rounding of either side. And batches of the smallest class (order
5, work areas larger than the order basis) against the same cells one by one.
"""
import numpy as np
import pytest

from celeris_b200 import capi
from oracle import rcwa as RO

pytestmark = pytest.mark.gpu

TOL = 1e-10  # the parity tolerance of the RCWA tests (relative to the fields, absolute for powers)

BASE = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=4.0, eps_bg=1.0, fill_x=0.55,
            thickness_um=0.6)


def check(cells):
    res, info = capi.rcwa_batch([capi.rcwa_cell(**c) for c in cells])
    assert not np.any(info)
    for i, c in enumerate(cells):
        for r, (ex, ey) in zip(res[2 * i:2 * i + 2], ((1.0, 0.0), (0.0, 1.0))):
            o = RO.solve_cell(**c, Ex0=ex, Ey0=ey)
            scale = max(abs(o["tx0"]), abs(o["ty0"]))
            for key in ("tx0", "ty0"):
                assert abs(r[key] - o[key]) <= TOL * scale, (key, r[key], o[key])
            for key in ("R", "T", "de_t0", "de_r0"):
                assert abs(r[key] - o[key]) <= TOL, (key, r[key], o[key])


@pytest.mark.parametrize("h,eps", [(5e-4, 4.0), (5e-4, complex(4.0, 0.3)), (7.0, complex(4.0, 0.01))])
@pytest.mark.parametrize("Mx,My,fill_y,shape", [(1, 1, 0.55, 0), (2, 1, 0.4, 0), (3, 3, 0.55, 0), (2, 4, 0.3, 0),
                                                (3, 3, 0.55, 1), (5, 5, 0.55, 0), (7, 7, 0.55, 0), (4, 3, 0.45, 3)])
def test_thin_and_thick(h, eps, Mx, My, fill_y, shape):
    check([dict(BASE, thickness_um=h, eps_pillar=eps, Mx=Mx, My=My, fill_y=fill_y, shape=shape, grid=128 if shape else 0)])


@pytest.mark.parametrize("h", [0.6, 5e-4])
@pytest.mark.parametrize("square", [True, False])
def test_smallest_classes_in_large_batches(h, square):
    cells = [dict(BASE, thickness_um=h, Mx=1, My=1, fill_x=0.2 + 0.0015 * i, fill_y=0.2 + 0.0015 * i if square else 0.4)
             for i in range(401)]
    res, info = capi.rcwa_batch([capi.rcwa_cell(**c) for c in cells])
    assert not np.any(info)
    for i in range(0, 401, 8):
        one, _ = capi.rcwa_batch([capi.rcwa_cell(**cells[i])])
        for a, b in zip(res[2 * i:2 * i + 2], one):
            for key in ("tx0", "ty0", "R", "T"):
                assert abs(a[key] - b[key]) <= TOL, (i, key, a[key], b[key])
