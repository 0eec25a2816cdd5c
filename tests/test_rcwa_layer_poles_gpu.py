"""Layers with a mode of larger q than sqrt(max |eps|) k0 (plasmon modes of negative
permittivities; an absorbing incident medium at oblique incidence), at thicknesses where that
mode's phase is a power of two times pi, so that sin(q x) = 0 in one of the layer's slabs.
Against the oracle at the RCWA tests' parity tolerance.
"""
import numpy as np
import pytest
import scipy.linalg as sla

from celeris_b200 import capi
from oracle import rcwa as RO

pytestmark = pytest.mark.gpu

TOL = 1e-10  # the parity tolerance of the RCWA tests (relative to the fields, absolute for powers)

METAL = dict(period_um=0.7025, wavelength_um=0.8944, n_inc=1.0, n_sub=1.46, eps_pillar=-4.0, eps_bg=2.25, fill_x=0.5577)
RASTER = dict(METAL, Mx=2, My=2, shape=capi.SHAPE_ELLIPSE, grid=64)
CELLS = {
    "one class": RASTER,
    "two classes": dict(RASTER, fill_y=0.5),
    "oblique": dict(METAL, Mx=2, My=1, theta_rad=0.3, phi_rad=0.4),
    "absorbing incident medium": dict(period_um=0.3, wavelength_um=0.633, n_inc=2.5j, n_sub=1.46, eps_pillar=2.5,
                                      eps_bg=2.25, fill_x=0.55, Mx=2, My=1, theta_rad=1.0, phi_rad=0.4),
}


def oracle_layer(c, thickness):
    return dict(eps_pillar=c["eps_pillar"], eps_bg=c["eps_bg"], fill_x=c["fill_x"], fill_y=c.get("fill_y", c["fill_x"]),
                thickness=thickness, shape=c.get("shape", 0), shape_param=0.5, rotation=0.0, grid=c.get("grid"))


def largest_q(c):
    """The largest real q of the layer's modes that the incident order meets."""
    seen = []

    def eig(a):
        seen.append(sla.eig(a))
        return seen[0]

    RO.solve(c["n_inc"], [oracle_layer(c, 0.1)], c["n_sub"], c["period_um"], c["period_um"], c["wavelength_um"],
             c.get("theta_rad", 0.0), c.get("phi_rad", 0.0), 1.0, 0.0, c["Mx"], c["My"], eig=eig)
    w, v = seen[0]
    q, n = np.sqrt(w + 0j), len(w) // 2
    met = np.abs(v[n // 2]) + np.abs(v[n + n // 2]) > 1e-6
    return float(np.abs(q[met & (np.abs(q.imag) < 1e-6 * np.abs(q))].real).max())


def compare(r, o):
    scale = max(abs(o["tx0"]), abs(o["ty0"]))
    for key in ("tx0", "ty0"):
        assert abs(r[key] - o[key]) <= TOL * scale, (key, r[key], o[key])
    for key in ("R", "T", "de_t0", "de_r0"):
        assert abs(r[key] - o[key]) <= TOL, (key, r[key], o[key])


@pytest.mark.parametrize("name", list(CELLS))
@pytest.mark.parametrize("m", [0, 1, 2, 3])
def test_at_the_pole(name, m):
    cell = dict(CELLS[name], thickness_um=np.pi / largest_q(CELLS[name]) * 2.0 ** m)
    res, info = capi.rcwa_batch([capi.rcwa_cell(**cell)])
    assert info[0] == 0
    for r, (ex, ey) in zip(res, ((1.0, 0.0), (0.0, 1.0))):
        compare(r, RO.solve_cell(**cell, Ex0=ex, Ey0=ey))


def test_metal_layer_of_a_stack():
    h = 2.0 * np.pi / largest_q(RASTER)
    layers = [dict(RASTER, thickness_um=h), dict(RASTER, eps_pillar=4.0, thickness_um=0.3)]
    got = capi.solve_rcwa_2d_stack([capi.rcwa_cell(**c) for c in layers], 1.0, 0.0)
    ol = [oracle_layer(c, c["thickness_um"]) for c in layers]
    c = layers[0]
    compare(got, RO.solve(c["n_inc"], ol, c["n_sub"], c["period_um"], c["period_um"], c["wavelength_um"], 0.0, 0.0, 1.0,
                          0.0, 2, 2))
