"""The residual of a state at rest with a constant field, which is zero (GPU).  Its only fluxes are the constants p + B^2/2 - B_n^2
and -B_n B_t; the node pairs' and the faces' are rounded alike, and div B is formed from differences, so that at p = 1
on elements of size 1, where every coefficient is a power of two, a constant cancels to the last bit.  Where a component of the
momentum collects two constants (B_x and B_y both nonzero), or at p = 2, 3, the sum's own roundings remain: at most
8 of terms whose coefficients sum to 18 x 2/h (D, 1/w), of the constant's size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("field", [(28.2094791773878, 0.0, 0.0), (0.0, 3.3, 0.0), (1.7, -0.9, 0.3), (0.1, 0.2, 11.1)])
def test_state_at_rest(pkg, p, field):
    nx, ny = 9, 7
    b2 = sum(f * f for f in field)
    w = np.array([1.1, 0.0, 0.0, 0.0, *field, 0.7 + 0.5 * b2])
    u = np.full((8, p + 1, p + 1, nx + 2, ny + 2), np.nan, order="F")
    u[...] = w[:, None, None, None, None]
    with pkg.DGSolver(nx, ny, p, 3, (0.0, float(nx), 0.0, float(ny)), 1.4) as g:
        g.upload_state(0, u)
        g.semidiscretize(1, 0)
        ut = g.download_ut(1)
    if p == 1 and field[0] * field[1] == 0.0:
        assert not ut.any(), np.abs(ut).reshape(8, -1).max(1)
    else:
        assert np.abs(ut).max() <= 8 * 0.5 * np.finfo(float).eps * 18 * 2 * 2 * b2  # two directions of size B^2 at most
