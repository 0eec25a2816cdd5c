"""Layers solved through their two-port (no eigendecomposition) at the sizes and
thicknesses where it can go wrong, through the C ABI: orders around the panel and lane
counts of its Gauss-Jordan solves, real and complex arithmetic, layers thin enough to
need no doubling and thick enough to need many, thicknesses at which a mode of the
layer makes a doubling singular, and the thicknesses that leave it for the
eigendecomposition. Against the oracle at the RCWA tests' parity tolerance, or against
the analytic slab.
"""
import numpy as np
import pytest

from celeris_b200 import capi
from oracle import rcwa as RO

pytestmark = pytest.mark.gpu

TOL = 1e-10  # the parity tolerance of the RCWA tests (relative to the fields, absolute for powers)

BASE = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=4.0, eps_bg=1.0, fill_x=0.55,
            thickness_um=0.6)


def check(cell):
    c = dict(BASE)
    c.update(cell)
    res, info = capi.rcwa_batch([capi.rcwa_cell(**c)])
    assert info[0] == 0
    for r, (ex, ey) in zip(res, ((1.0, 0.0), (0.0, 1.0))):
        o = RO.solve_cell(**c, Ex0=ex, Ey0=ey)
        scale = max(abs(o["tx0"]), abs(o["ty0"]))
        for key in ("tx0", "ty0"):
            assert abs(r[key] - o[key]) <= TOL * scale, (key, r[key], o[key])
        for key in ("R", "T", "de_t0", "de_r0"):
            assert abs(r[key] - o[key]) <= TOL, (key, r[key], o[key])


OBL = dict(theta_rad=0.2, phi_rad=0.5, period_x_um=0.42, period_y_um=0.38, fill_y=0.4)


@pytest.mark.parametrize("Mx,My", [(0, 0), (1, 0), (0, 3), (1, 1), (1, 2), (1, 3), (2, 2), (1, 5), (3, 2), (3, 4),
                                   (4, 4), (4, 6), (5, 6)])
def test_orders_oblique(Mx, My):
    check(dict(OBL, Mx=Mx, My=My))


@pytest.mark.parametrize("Mx,My", [(1, 1), (2, 1), (2, 2), (2, 3), (3, 3), (4, 4), (5, 4), (7, 7), (8, 8)])
def test_orders_parity_classes(Mx, My):
    check(dict(Mx=Mx, My=My, fill_y=0.55 if Mx == My else 0.4))


@pytest.mark.parametrize("extra", [dict(eps_pillar=complex(6.0, 0.3)), dict(eps_pillar=complex(-2.0, 1.5), thickness_um=0.08),
                                   dict(eps_bg=complex(1.2, 0.01)), dict(n_sub=complex(1.5, 0.2))])
@pytest.mark.parametrize("oblique", [False, True])
def test_lossy(extra, oblique):
    check(dict(OBL if oblique else {}, Mx=3, My=3, **extra))


@pytest.mark.parametrize("h", [1e-4, 9e-4, 2e-3, 0.02, 0.1, 1.7, 4.5, 7.0])
def test_thicknesses(h):
    # below 0.01 / k0 = 1.0e-3 um and above 100 rad (5.04 um at n = 2) through the eigendecomposition
    check(dict(Mx=2, thickness_um=h))
    check(dict(OBL, Mx=2, My=1, thickness_um=h))


@pytest.mark.parametrize("waves", [0.5, 1.0, 2.0, 4.0, 8.0, 1.5, 3.0])
@pytest.mark.parametrize("n_layer", [1.46, 2.0])
def test_uniform_layer_at_its_poles(waves, n_layer):
    """A uniform layer of a whole number of half-waves: cos(q h / 2^j) = 0 exactly for the
    normal-incidence mode at one of the doublings. The Airy formula is the reference."""
    wl, ni, ns = 0.633, 1.0, 1.46
    h = waves * wl / n_layer
    c = dict(BASE, n_inc=ni, n_sub=ns, eps_pillar=n_layer ** 2, eps_bg=n_layer ** 2, fill_x=0.5, thickness_um=h, Mx=2)
    r12, r23 = (ni - n_layer) / (ni + n_layer), (n_layer - ns) / (n_layer + ns)
    e = np.exp(2j * np.pi * n_layer * h / wl)
    r = (r12 + r23 * e * e) / (1 + r12 * r23 * e * e)
    res, info = capi.rcwa_batch([capi.rcwa_cell(**c)])
    assert info[0] == 0
    for q in res:
        assert abs(q["R"] - abs(r) ** 2) <= TOL
        assert abs(q["T"] - (1 - abs(r) ** 2)) <= TOL


def test_pole_in_a_stack_layer_and_redo_in_a_batch():
    """Half-wave layers inside a stack, against the oracle; and a batch in which only some
    cells meet a pole gives the same as the cells alone."""
    wl = 0.633
    layers = [dict(BASE, Mx=2, eps_pillar=4.0, eps_bg=4.0, thickness_um=wl / 4.0), dict(BASE, Mx=2, thickness_um=0.31)]
    got = capi.solve_rcwa_2d_stack([capi.rcwa_cell(**c) for c in layers], 1.0, 0.0)
    ol = [dict(eps_pillar=c["eps_pillar"], eps_bg=c["eps_bg"], fill_x=c["fill_x"], fill_y=c["fill_x"],
               thickness=c["thickness_um"], shape=0, shape_param=0.5, rotation=0.0) for c in layers]
    o = RO.solve(1.0, ol, 1.46, 0.4, 0.4, wl, 0.0, 0.0, 1.0, 0.0, 2, 2)
    assert abs(got["tx0"] - o["tx0"]) <= TOL * abs(o["tx0"])
    assert abs(got["R"] - o["R"]) <= TOL
    cells = [dict(BASE, Mx=2, eps_pillar=e, eps_bg=e, thickness_um=wl / 2.0) for e in (4.0, 2.25, 4.0, 3.0)]
    cells += [dict(BASE, Mx=2, thickness_um=h) for h in (0.2, 0.4)]
    res, info = capi.rcwa_batch([capi.rcwa_cell(**c) for c in cells])
    assert not np.any(info)
    for i, c in enumerate(cells):
        one, _ = capi.rcwa_batch([capi.rcwa_cell(**c)])
        assert abs(res[2 * i]["tx0"] - one[0]["tx0"]) <= TOL


@pytest.mark.parametrize("shape", [capi.SHAPE_RECT, capi.SHAPE_ELLIPSE, capi.SHAPE_CROSS, capi.SHAPE_RING])
@pytest.mark.parametrize("grid,Mx,My,fx,fy,param", [
    (128, 2, 2, 0.55, 0.55, 0.5), (100, 2, 1, 0.6, 0.35, 0.4), (37, 1, 3, 0.31, 0.77, 0.3), (3, 2, 2, 0.7, 0.7, 0.5),
    (64, 3, 2, 1.0, 1.0, 0.9), (48, 2, 2, 1.3, 0.5, 1.2), (33, 2, 2, 0.5, 0.5, 0.0), (256, 1, 1, 1e-3, 0.6, 0.5),
])
def test_raster_sample_intervals(shape, grid, Mx, My, fx, fy, param):
    """Parity-class operators of rasterised shapes from sample intervals and prefix sums:
    odd and tiny rasters (an order a multiple of the raster size), fills of nothing and of
    more than the cell, cross and ring parameters of 0 and above 1."""
    eps_p = complex(5.0, 0.1) if grid == 100 else 5.0
    cell = dict(Mx=Mx, My=My, shape=shape, grid=grid, force_laurent=1, fill_x=fx, fill_y=fy, shape_param=param,
                eps_pillar=eps_p)
    eps = RO.rasterize_eps(eps_p, 1.0, grid, grid, shape, fx, fy, param, 0.0)
    if np.linalg.cond(RO.laurent_toeplitz(eps, grid, grid, Mx, My)) > 1e12:
        # fewer raster points than orders: the Laurent matrix is singular and no solution
        # is defined (the oracle's inverse raises or is rounding noise); the call returns
        _, info = capi.rcwa_batch([capi.rcwa_cell(**dict(BASE, **cell))])
        assert info.shape == (1,)
    elif np.ptp(eps.real) == 0.0 and np.ptp(eps.imag) == 0.0:
        # the shape covers nothing or everything: a uniform layer, whose degenerate
        # eigenvectors leave the oracle's numbers undefined; the Airy formula holds
        n1, h = np.sqrt(eps[0, 0] + 0j), BASE["thickness_um"]
        r12, r23 = (1.0 - n1) / (1.0 + n1), (n1 - 1.46) / (n1 + 1.46)
        e2 = np.exp(4j * np.pi * n1 * h / BASE["wavelength_um"])
        R = abs((r12 + r23 * e2) / (1 + r12 * r23 * e2)) ** 2
        res, info = capi.rcwa_batch([capi.rcwa_cell(**dict(BASE, **cell))])
        assert info[0] == 0
        assert all(abs(q["R"] - R) <= TOL for q in res)
    else:
        check(cell)
