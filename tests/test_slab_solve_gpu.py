"""The block elimination of the RCWA layers on its own, against numpy: orders around its
panel (16), lane (32, 64, 128, 256) and warp counts, in both block sizes, real and
complex, with and without the inverse.
"""
import ctypes

import numpy as np
import pytest

from celeris_b200 import capi

pytestmark = pytest.mark.gpu

U = np.finfo(np.float64).eps / 2
P = ctypes.POINTER(ctypes.c_double)


def solve(a, b, inverse=False, threads=512, lost_warp=-1):
    """(ok, x, ainv) of a x = b through celeris_debug_slab_solve."""
    n, nrhs, cplx = a.shape[0], b.shape[1], np.iscomplexobj(a)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    x, inv, ok = np.zeros_like(b), np.zeros_like(a), ctypes.c_int(-1)
    ptr = lambda v: v.ctypes.data_as(P)  # noqa: E731
    capi.check(capi.load().celeris_debug_slab_solve(n, nrhs, int(cplx), int(inverse), threads, lost_warp, ptr(a), ptr(b),
                                                    ptr(x), ptr(inv), ctypes.byref(ok)))
    return ok.value, x, inv


def unitary(n, cplx, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n))
    if cplx:
        a = a + 1j * rng.standard_normal((n, n))
    return np.linalg.qr(a)[0]


@pytest.mark.parametrize("n", [1, 2, 5, 15, 16, 17, 31, 32, 33, 49, 61, 64, 65, 98, 127, 128, 129, 162, 255, 256, 257,
                               481, 512])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("threads", [256, 512])
def test_elimination(n, cplx, threads):
    """A handed-over column that is read before all of it is written shows here as a wrong
    solution. Unitary matrices (condition 1): Gauss-Jordan's forward error is within 2 n u times the
    growth of the pivots, taken as n."""
    if threads == 256 and n > 256:
        pytest.skip("orders above 256 take sixteen warps")
    a = unitary(n, cplx, n)
    tol = 2.0 * (n + 4) ** 2 * U
    for nrhs, inverse in ((1, False), (n, True), (2, True)):
        b = unitary(max(n, nrhs), cplx, 7 * n + nrhs)[:n, :nrhs]
        ok, x, inv = solve(a, b, inverse, threads)
        assert ok == 1
        want = a.conj().T @ b
        assert np.linalg.norm(x - want) <= tol * np.linalg.norm(want)
        if inverse:
            assert np.linalg.norm(inv - a.conj().T) <= tol * np.sqrt(n)


@pytest.mark.parametrize("warp", [0, 1, 3, 7])
@pytest.mark.parametrize("cplx", [False, True])
def test_a_warp_that_gives_up_is_reported(warp, cplx):
    """One warp's wait runs out while the others' do not (order 1: one column, whose owner, warp
    0, hands it over before it waits). The elimination reports it, from whichever warp: that warp's
    columns are missing from the update."""
    a = unitary(1, cplx, 1)
    ok, x, _ = solve(a, a, lost_warp=warp)
    assert ok == 0 and not np.any(x)
    assert solve(a, a)[0] == 1


@pytest.mark.parametrize("n,col", [(1, 0), (5, 2), (5, 4), (9, 3), (9, 8), (17, 16), (25, 7), (33, 20), (61, 40), (100, 99),
                                   (162, 17), (300, 299)])
@pytest.mark.parametrize("cplx", [False, True])
def test_a_column_without_a_pivot_writes_nothing_outside(n, col, cplx):
    """A zero column ends the elimination, and the row its search falls on, which may lie past the
    matrix, is not recorded (the call checks the neighbouring arrays and reports an error)."""
    a = unitary(n, cplx, n)
    a[:, col] = 0.0
    ok, x, _ = solve(a, unitary(n, cplx, n)[:, :1])
    assert ok == 0 and not np.any(x)


@pytest.mark.parametrize("n", [1, 7, 33, 98])
@pytest.mark.parametrize("threads", [256, 512])
def test_block_maxima_keep_nan(n, threads):
    """One NaN among numbers shows in the norm and in the largest entry, wherever it lies."""
    a = np.random.default_rng(n).standard_normal((n, n))
    out = np.zeros(2)

    def maxima(m):
        capi.check(capi.load().celeris_debug_slab_max(n, threads, m.ctypes.data_as(P), out.ctypes.data_as(P)))
        return out.copy()

    got = maxima(a)
    assert abs(got[0] - np.abs(a).sum(axis=1).max()) <= 2 * n * U * got[0] and got[1] == np.abs(a).max()
    for e in {0, n * n // 3, n * n - 1}:
        b = a.copy()
        b.flat[e] = np.nan
        assert np.all(np.isnan(maxima(b)))
