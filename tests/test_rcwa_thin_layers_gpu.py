"""Thin layers keep the eigendecomposition's digits: tx0 and ty0 of both excitations against
values from 50-digit arithmetic on the FP64 layer operators (mpmath: the layer's cos and sin
series, doublings and the interface systems), relative to the largest field. Tolerance: 2 N u, the
order of the systems times the unit roundoff.
"""
import numpy as np
import pytest

from celeris_b200 import capi

pytestmark = pytest.mark.gpu

U = np.finfo(np.float64).eps / 2

NORMAL = dict(period_um=0.4, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=5.3, eps_bg=1.0, fill_x=0.45, fill_y=0.7,
              Mx=2, My=1)
OBLIQUE = dict(NORMAL, Mx=1, theta_rad=0.3, phi_rad=0.7)

CASES = [
    (NORMAL, 0.0012, [0.8128818792581306 + 0.014300932246442133j, 0, 0, 0.8128802193659889 + 0.014381380250169946j]),
    (NORMAL, 0.0025, [0.8124625009324392 + 0.029734904705840906j, 0, 0, 0.8124508779187793 + 0.030005205674509036j]),
    (NORMAL, 0.005, [0.8108430430733217 + 0.059233799360224194j, 0, 0, 0.8107634727781604 + 0.06015746153894843j]),
    (NORMAL, 0.039, [0.6934333797419572 + 0.4261261012037453j, 0, 0, 0.6687701205811242 + 0.45717807546022843j]),
    (OBLIQUE, 0.0012, [0.8144200309903993 + 0.013197781199533814j, -0.024993033531209945 - 0.0004817099724053033j,
                       0.5511536848043173 + 0.010638540890073746j, -18.1490854809383 - 0.31340950826133157j]),
    (OBLIQUE, 0.0025, [0.8140420012235076 + 0.027481145137415612j, -0.02497989502121838 - 0.000999574073504204j,
                       0.5508895796315818 + 0.022111313212704237j, -18.138592478509906 - 0.6541288690160095j]),
    (OBLIQUE, 0.005, [0.8125731401028312 + 0.05488743575051568j, -0.024930704434801765 - 0.001982743485550424j,
                      0.5498890672973435 + 0.04399538906250213j, -18.097232755269868 - 1.3121043812699562j]),
    (OBLIQUE, 0.039, [0.7027555483414798 + 0.40250820352705197j, -0.02256136377148199 - 0.01375624801657834j,
                      0.4965978630986682 + 0.31136389806250814j, -14.669841531253832 - 9.749054481344407j]),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("as_stack", [False, True])
def test_thin_layer(case, as_stack):
    base, h, want = CASES[case]
    cell = capi.rcwa_cell(**dict(base, thickness_um=h))
    res, info = capi.rcwa_stack_batch([[cell]]) if as_stack else capi.rcwa_batch([cell])
    assert info[0] == 0
    got = np.array([res[0]["tx0"], res[0]["ty0"], res[1]["tx0"], res[1]["ty0"]])
    tol = 2 * (2 * base["Mx"] + 1) * (2 * base["My"] + 1) * U
    assert np.abs(got - np.array(want)).max() <= tol * np.abs(want).max()
