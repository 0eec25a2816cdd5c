"""The FP64 far-field sums (field and adjoint) at the edges of their tiles and of
their domain: pillar and pixel counts around the thread strips, chunks and tiles,
and inputs that leave the table form's domain (coordinates, wavenumber, z), where
the direct form runs. Against the oracle.

Tolerance: the phase k R of a term is rounded to half an ulp of k R on either side
and R itself to about an ulp, so a term's phase differs by at most ~4 eps k R; the
amplitude, sine and cosine and the sums add some tens of eps. Both are counted
without cancellation: |dE| <= (6 eps k R_max + 64 eps) sum_j |t_j| / R_min.
"""
import numpy as np
import pytest

from celeris_b200 import capi
from oracle import farfield as F

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


def inputs(npil, seed, scale=8.0):
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(-scale, scale, npil), rng.uniform(-scale, scale, npil)
    t = rng.uniform(0.0, 1.0, npil) * np.exp(1j * rng.uniform(0, 2 * np.pi, npil))
    t[:: max(1, npil // 3)] = 0.0  # exact zeros
    return x, y, t


def tolerance(x, y, z, k, amp, W):
    far = np.hypot(np.abs(x).max() + W, np.abs(y).max() + W)
    rmax = np.hypot(far, z)
    rmin = abs(z) if z != 0.0 else 0.05
    return (6 * EPS * abs(k) * rmax + 64 * EPS) * amp / rmin


@pytest.mark.parametrize("npil,n", [(1, 1), (1, 2), (31, 3), (32, 4), (33, 5), (63, 16), (64, 17), (255, 31),
                                    (256, 33), (257, 64), (1009, 41), (4096, 65), (9001, 127)])
def test_field_and_adjoint_sizes(npil, n):
    import torch

    from celeris_b200 import torch_ops as T

    x, y, t = inputs(npil, npil + n)
    z, wl, W = 30.0, 0.55, 3.0
    if n == 1:  # a one-pixel grid has no step: the reference's expression gives NaN there
        n = 2
    grid = T.FarFieldGrid(n, W, z, wl, 0.3, -0.2)
    E, _, _ = capi.rs_field(x, y, t, 0.3, -0.2, z, grid.k, n, W)
    Eo = F.rs_field(x, y, t, 0.3, -0.2, z, grid.k, n, W)
    assert np.max(np.abs(E - Eo)) <= tolerance(x, y, z, grid.k, np.abs(t).sum(), W + 0.3)
    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    v[0, :] = 0.0
    out = T.rs_adjoint_dev(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"),
                           torch.tensor(v, device="cuda"), grid).cpu().numpy()
    ref = F.rs_adjoint(x, y, grid.cx, grid.cy, z, grid.k, n, W, v)
    assert np.max(np.abs(out - ref)) <= tolerance(x, y, z, grid.k, np.abs(v).sum(), W + 0.3)


@pytest.mark.parametrize("name", ["far_pillar", "far_pixels", "short_wave", "negative_k", "zero_z", "far_z", "zero_k"])
def test_outside_the_table_forms_domain(name):
    x, y, t = inputs(301, 5)
    cx, z, wl, W, n = 0.0, 30.0, 0.55, 3.0, 13
    k = 2 * np.pi / wl
    if name == "far_pillar":
        x[70] = 3e9
    elif name == "far_pixels":
        cx = 5e9
    elif name == "short_wave":
        k = 5e3
    elif name == "negative_k":
        k = -k
    elif name == "zero_z":
        z = 0.0
        x = np.abs(x) + 3.05  # off the pixels
    elif name == "far_z":
        z = 2e9
    elif name == "zero_k":
        k = 0.0
    E, _, _ = capi.rs_field(x, y, t, cx, 0.0, z, k, n, W)
    Eo = F.rs_field(x, y, t, cx, 0.0, z, k, n, W)
    assert np.all(np.isfinite(E.view(float)))
    assert np.max(np.abs(E - Eo)) <= tolerance(x - cx, y, z, k, np.abs(t).sum(), W)
