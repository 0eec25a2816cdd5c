"""Device memory of RCWA batches in the order basis: the arena that a batch grows from nothing, against
the matrices an eigendecomposition of the same batch holds (9.75 n^2 complex a cell; 7.75 n^2 a layer
and 7 n^2 a stack; arenas grow by a quarter more than asked), and sets with more layers than run at a time against the same stacks alone.
"""
import numpy as np
import pytest
import torch

from celeris_b200 import capi

pytestmark = pytest.mark.gpu

BASE = dict(period_x_um=0.4, period_y_um=0.38, wavelength_um=0.633, n_inc=1.0, n_sub=1.46, eps_pillar=4.0, eps_bg=1.0,
            fill_x=0.5, fill_y=0.6, thickness_um=0.4)


def grown(call):
    """Device bytes that `call` leaves allocated, from an empty workspace."""
    call()  # modules, tuning and graph memory
    capi.check(capi.load().celeris_release_workspace())
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    call()
    return before - torch.cuda.mem_get_info()[0]


def square(M):
    return 16.0 * (2 * (2 * M + 1) ** 2) ** 2


def test_cells():
    cells = [capi.rcwa_cell(**dict(BASE, Mx=4, theta_rad=0.2, fill_x=0.3 + 0.002 * i)) for i in range(256)]
    assert grown(lambda: capi.rcwa_batch(cells)) <= 1.25 * 256 * 9.75 * square(4) + (32 << 20)


@pytest.mark.parametrize("layers", [1, 2])
def test_stacks(layers):
    stacks = [[capi.rcwa_cell(**dict(BASE, Mx=4, fill_x=0.3 + 0.002 * i, thickness_um=0.2 + 0.1 * k)) for k in range(layers)]
              for i in range(128)]
    assert grown(lambda: capi.rcwa_stack_batch(stacks)) <= 1.25 * 128 * (7.75 * layers + 7.0) * square(4) + (32 << 20)


def test_more_layers_than_run_at_a_time():
    """1400 layers, rasterised and analytic ones mixed, in stacks of seven."""
    def stack(i):
        return [capi.rcwa_cell(**dict(BASE, Mx=1, fill_x=0.3 + 0.002 * i, thickness_um=0.1 + 0.05 * k, shape=(i + k) % 2,
                                      grid=32 if (i + k) % 2 else 0)) for k in range(7)]

    stacks = [stack(i) for i in range(200)]
    assert 7 * len(stacks) > 8 * torch.cuda.get_device_properties(0).multi_processor_count
    res, info = capi.rcwa_stack_batch(stacks)
    assert not np.any(info)
    for i in (0, 1, 99, 168, 169, 170, 199):
        one, _ = capi.rcwa_stack_batch([stacks[i]])
        for a, b in zip(res[2 * i:2 * i + 2], one):
            for key in ("tx0", "ty0", "R", "T"):
                assert abs(a[key] - b[key]) <= 1e-10, (i, key, a[key], b[key])
