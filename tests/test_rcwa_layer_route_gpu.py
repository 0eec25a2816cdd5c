"""Which thick layers go through the eigendecomposition (where leaving out doublings would cost more
than it), read off the kernels of a batch, and both sides of each line against the oracle at the
RCWA tests' parity tolerance (layers that absorb a little, so that no resonance amplifies
rounding).
"""
import numpy as np
import pytest

from celeris_b200 import capi
from oracle import rcwa as RO

pytestmark = pytest.mark.gpu

TOL = 1e-10
BASE = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_bg=1.0, fill_x=0.55)


def thickness(phase, eps):
    return phase * BASE["wavelength_um"] / (2.0 * np.pi * np.sqrt(abs(eps)))


def launches(cell):
    lib, arr = capi.load(), [capi.rcwa_cell(**cell)]
    for _ in range(2):
        before = lib.celeris_launch_count()
        _, info = capi.rcwa_batch(arr)
        assert info[0] == 0
    return lib.celeris_launch_count() - before


@pytest.mark.parametrize("phase,two_port", [(30.0, True), (47.0, True), (51.0, False), (90.0, False)])
@pytest.mark.parametrize("oblique", [False, True])
def test_route_by_phase(phase, two_port, oblique):
    cell = dict(BASE, eps_pillar=4.0, Mx=2, thickness_um=thickness(phase, 4.0), **(dict(theta_rad=0.3) if oblique else {}))
    fast, slow = (3, 8) if oblique else (4, 7)
    assert launches(cell) == (fast if two_port else slow)


@pytest.mark.parametrize("M,eps,phase,two_port", [(11, 4.0, 20.0, True), (11, 4.0, 30.0, False), (11, 4.0 + 0.01j, 10.0, True),
                                                  (11, 4.0 + 0.01j, 20.0, False)])
def test_route_of_large_classes(M, eps, phase, two_port):
    assert launches(dict(BASE, eps_pillar=eps, Mx=M, thickness_um=thickness(phase, eps))) == (4 if two_port else 7)


@pytest.mark.parametrize("phase", [23.0, 47.0, 51.0])
@pytest.mark.parametrize("extra", [dict(Mx=3), dict(Mx=2, My=1, fill_y=0.4), dict(Mx=2, My=1, theta_rad=0.3, phi_rad=0.4)])
def test_thick_layers_against_the_oracle(phase, extra):
    eps = 4.0 + 0.02j
    cell = dict(BASE, eps_pillar=eps, thickness_um=thickness(phase, eps), **extra)
    res, info = capi.rcwa_batch([capi.rcwa_cell(**cell)])
    assert info[0] == 0
    for r, (ex, ey) in zip(res, ((1.0, 0.0), (0.0, 1.0))):
        o = RO.solve_cell(**cell, Ex0=ex, Ey0=ey)
        scale = max(abs(o["tx0"]), abs(o["ty0"]))
        for key in ("tx0", "ty0"):
            assert abs(r[key] - o[key]) <= TOL * scale, (key, r[key], o[key])
        for key in ("R", "T", "de_t0", "de_r0"):
            assert abs(r[key] - o[key]) <= TOL, (key, r[key], o[key])
