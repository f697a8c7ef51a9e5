"""The identities by which the residual kernel (csrc/residual.cuh) leaves out terms of the reference's
sum (CPU, on the library's GLL tables)."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("p", [1, 2, 3])
def test_own_flux_of_a_node_cancels(pkg, p):
    """the flux differencing's diagonal 2 D_kk is zero inside the element and 1/w at its ends, so it
    cancels the own-flux part of the surface terms; a row of D sums to zero, so a constant may be
    left out of all fluxes of a line"""
    n = p + 1
    w, D = np.zeros(n), np.zeros((n, n), order="F")
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert pkg.capi.load().mhd_gpu_gll_tables(p, None, ptr(w), None, None, ptr(D), None, None) == 0
    eps = np.finfo(float).eps
    assert abs(2 * D[0, 0] * w[0] + 1) <= eps and abs(2 * D[p, p] * w[p] - 1) <= eps
    assert np.all(np.diag(D)[1:-1] == 0.0)
    assert np.abs(D.sum(1)).max() <= n * eps * np.abs(D).max()
